"""The branches that a call's sizes choose, at the sizes where each can go wrong: tails of tiles, half-empty head pairs,
cut sequences, short runs, strided operands.  Tolerances as in ``test_ssd_gpu``: 2e-2 for 16-bit types (P and the state
copy are rounded to 16 bits, 2^-8, and sums of N(0,1) products average that out), 1e-4 for fp32."""
import pytest
import torch

from oracle import ssd_oracle as O

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _no_device_side_timeouts():
    yield
    if torch.cuda.is_available():
        import workloadsuite_b200 as W

        assert W.device_status(DEV) == 0


def _check(inp, kernel, tol, dt=None, D=None, z=None, **kw):
    import workloadsuite_b200 as W

    d = {k: v.to(DEV) for k, v in inp.items()}
    dev = lambda t: None if t is None else t.to(DEV)
    Y, H = W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, dt=dev(dt), initial_states=d.get("initial_states"),
                         return_final_state=True, D=dev(D), z=dev(z), kernel=kernel, **kw)
    torch.cuda.synchronize()
    Yr, Hr = O.ssd_recurrence(inp["X"], inp["A"], inp["B"], inp["C"], dt=dt, initial_states=inp.get("initial_states"),
                              return_final_state=True)
    if D is not None:
        Yr = Yr + inp["X"].double() * D.double()[None, None, :, None]
    if z is not None:
        Yr = Yr * torch.nn.functional.silu(z.double())
    assert max(O.error_metrics(Y.cpu(), Yr)) < tol
    assert ((H.cpu().double() - Hr).abs().amax(dim=(2, 3)) / Hr.abs().amax(dim=(2, 3)).clamp_min(1e-30)).max().item() < tol


@pytest.mark.parametrize("s", [1, 31, 127, 128, 129, 300])
@pytest.mark.parametrize("h,g,n", [(3, 1, 128), (4, 2, 64), (5, 5, 64)])
def test_tensor_core_kernel_takes_any_length_and_odd_heads(s, h, g, n):
    """Tails that are no whole tile (zero-filled by TMA, clipped on the way out) and groups whose last pair of heads is
    half empty, with and without skip and gate."""
    inp = O.make_inputs(b=2, s=s, h=h, p=64, n=n, g=g, dtype=torch.bfloat16, init=True, seed=60 + s, decay_scale=0.1)
    gen = torch.Generator().manual_seed(s)
    dt = (0.5 + torch.rand(2, s, h, generator=gen)).bfloat16()
    _check(inp, "tcgen05", 2e-2, dt=dt)
    D, z = torch.randn(h, generator=gen).bfloat16(), torch.randn(2, s, h, 64, generator=gen).bfloat16()
    _check(inp, "tcgen05", 2e-2, dt=dt, D=D, z=z)


@pytest.mark.parametrize("dtype,ulp", [(torch.bfloat16, 2 ** -7), (torch.float16, 2 ** -10)])
@pytest.mark.parametrize("h,g", [(3, 1), (4, 4), (10, 2)])
def test_groups_with_an_odd_number_of_heads_round_the_decayed_x_once(h, g, dtype, ulp):
    """A rounding's relative error is ulp / 2 / sqrt(3) * 0.72 in the mean (the 0.72 for mantissas spread over their octave): 0.21
    ulp.  The final state sums once-rounded products, so that is its error too (0.29 with the scale rounded as well); Y has
    P, the state's copy and its own rounding, and the gate in fp32 between two roundings (0.38 against 0.48 with a packed gate)."""
    import workloadsuite_b200 as W

    inp = O.make_inputs(b=2, s=1024, h=h, p=64, n=128, g=g, dtype=dtype, seed=66, decay_scale=1.0)
    d = {k: v.to(DEV) for k, v in inp.items()}
    gen = torch.Generator().manual_seed(67)
    D, z = torch.randn(h, generator=gen).to(dtype), torch.randn(2, 1024, h, 64, generator=gen).to(dtype)
    Y, H = W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 128, D=D.to(DEV), z=z.to(DEV), return_final_state=True)
    Yr, Hr = O.ssd_recurrence(inp["X"], inp["A"], inp["B"], inp["C"], return_final_state=True)
    Yr = (Yr + inp["X"].double() * D.double()[:, None]) * torch.nn.functional.silu(z.double())
    assert ((H.cpu().double() - Hr).norm() / Hr.norm()).item() < 0.24 * ulp
    assert ((Y.cpu().double() - Yr).norm() / Yr.norm()).item() < 0.42 * ulp


@pytest.mark.parametrize("dtype,eps", [(torch.bfloat16, 2 ** -8), (torch.float16, 2 ** -11)])
@pytest.mark.parametrize("s,h,g", [(20, 4, 1), (300, 4, 2), (130, 5, 1)])
def test_lengths_that_are_no_whole_tiles_are_rounded_once(s, h, g, dtype, eps):
    """Without a choice of kernel they are computed in fp32: Y is off by its own rounding (half an ulp, eps / 2 of the value
    and at most eps of it) and the fp32 sums' 1e-5, the fp32 final state by 1e-5."""
    import workloadsuite_b200 as W

    inp = O.make_inputs(b=2, s=s, h=h, p=64, n=128, g=g, dtype=dtype, init=True, seed=65 + s, decay_scale=0.1)
    dt = (0.5 + torch.rand(2, s, h, generator=torch.Generator().manual_seed(s))).to(dtype)
    d = {k: v.to(DEV) for k, v in inp.items()}
    Y, H = W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, dt=dt.to(DEV), initial_states=d["initial_states"],
                         return_final_state=True)
    Yr, Hr = O.ssd_recurrence(inp["X"], inp["A"], inp["B"], inp["C"], dt=dt, initial_states=inp["initial_states"],
                              return_final_state=True)
    assert ((Y.cpu().double() - Yr).abs() <= eps * Yr.abs() + 1e-5 * Yr.abs().max()).all()
    assert ((H.cpu().double() - Hr).abs().max() / Hr.abs().max()).item() < 1e-5


def _strong_decays(A, dt, case):
    """Puts decays into A [b,s,h] (and dt) that no run of factors can carry in 32 bits, differently in every head."""
    b, s, h = A.shape
    for k in range(h):
        if case == "every_token":
            A[:, :, k] = -30.0 - 7 * k
        elif case == "one_token":
            A[:, 5 + k::37, k] = -100.0
        elif case == "reset":
            A[:, 8 + k::41, k] = -float("inf")
        elif case == "far":
            A[:, 3 + k::29, k] = -1e30
        elif case == "idle_tokens":        # dt = 0, then strong decays
            A[:, 1::4, k], A[:, 2::4, k], A[:, 3::4, k] = -16.0, -16.0, -16.0
            dt[:, k % 4::4, k] = 0.0
        elif case == "steps_of_both_signs":
            dt[:, k::5, k] *= -1.0
        elif case == "tiny_steps":
            dt[:, k::3, k] = 2.0 ** -14


@pytest.mark.parametrize("s,h,g", [(128, 4, 1), (384, 4, 2), (300, 4, 1), (256, 5, 1)])
@pytest.mark.parametrize("case", ["every_token", "one_token", "reset", "far", "idle_tokens", "steps_of_both_signs", "tiny_steps"])
def test_decays_beyond_the_range_of_a_factor(case, s, h, g):
    """Factors of P that differ by more than 32-bit numbers can between neighbouring tokens: a strong decay in every token, in
    single ones at each place of a group of four, resets, dt = 0 and dt < 0.  Weights that survive must be there (the
    diagonal above all), Y and the states finite, the sum of the log-decays as given."""
    import workloadsuite_b200 as W

    inp = O.make_inputs(b=2, s=s, h=h, p=64, n=64, g=g, dtype=torch.bfloat16, init=True, seed=72, decay_scale=0.05)
    dt = (0.5 + torch.rand(2, s, h, generator=torch.Generator().manual_seed(73))).bfloat16()
    _strong_decays(inp["A"], dt, case)
    for kernel in ("tcgen05", "scan_f32"):
        _check(inp, kernel, 2e-2, dt=dt)
    _check(inp, "tcgen05", 2e-2, dt=dt, nsegments=2)
    d = {k: v.to(DEV) for k, v in inp.items()}
    _, ld = W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, dt=dt.to(DEV), kernel="tcgen05", return_logdecay=True)
    assert torch.allclose(ld.cpu().double(), O.total_logdecay(inp["A"]), rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("dtype,eps", [(torch.bfloat16, 2 ** -8), (torch.float16, 2 ** -11)])
@pytest.mark.parametrize("b,s,h,n", [(2, 300, 4, 64), (1, 3001, 4, 128)], ids=["whole", "lookback"])
@pytest.mark.parametrize("case", ["every_token", "one_token", "reset", "far", "idle_tokens", "steps_of_both_signs", "tiny_steps"])
def test_strong_decays_at_fp32_precision(case, b, s, h, n, dtype, eps):
    """The same where the library chooses and the length is no whole tiles: Y off by its own rounding and the fp32 sums' 1e-5, the
    state by 1e-6 (a sum over the few tokens that such decays leave), the sum of the log-decays rounded once."""
    import workloadsuite_b200 as W

    inp = O.make_inputs(b=b, s=s, h=h, p=64, n=n, g=1, dtype=dtype, init=True, seed=74, decay_scale=0.05)
    inp["A"].abs_().neg_()
    dt = (0.5 + torch.rand(b, s, h, generator=torch.Generator().manual_seed(75))).to(dtype)
    _strong_decays(inp["A"], dt, case)
    d = {k: v.to(DEV) for k, v in inp.items()}
    plan = W.plan(d["X"], d["A"], d["B"], d["C"], 1)
    assert plan["kernel"] == "scan_f32" and plan["launches"] == 2      # on the tensor cores, and the recurrence behind them
    Y, H, ld = W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, dt=dt.to(DEV), initial_states=d["initial_states"],
                             return_final_state=True, return_logdecay=True)
    Yr, Hr = O.ssd_recurrence(inp["X"], inp["A"], inp["B"], inp["C"], dt=dt, initial_states=inp["initial_states"],
                              return_final_state=True)
    assert ((Y.cpu().double() - Yr).abs() <= eps * Yr.abs() + 1e-5 * Yr.abs().max()).all()
    assert ((H.cpu().double() - Hr).norm() / Hr.norm()).item() < 1e-6
    assert torch.allclose(ld.cpu().double(), inp["A"].double().sum(1), rtol=2 ** -23, atol=0)


@pytest.mark.parametrize("resets", [1, 8, 20])
@pytest.mark.parametrize("decay", [-float("inf"), -100.0, -20.0])
def test_weights_behind_strong_decays_are_those_of_their_own_exponents(decay, resets):
    """One token with an x right behind tokens of strong decay: Y of the tokens after it is x (C.B) exp(mild decays), whatever
    came before.  What the 32 768 elements of a token are off by in the mean, from the exact value rounded to fp16, is the error
    of the weight (an approximate exponential's 2^-22 and four products' 2^-24: 5e-7) and of C.B (64 products in four accumulations,
    each of which cuts off up to 2^-23: 5e-7; one more in P.X), 1.1e-6, and what the elements add that it rounds the other way: a step
    of 7e-4 in 1.1e-6 / 7e-4 of them, 51, whose spread leaves 1.5e-7; three times that."""
    import workloadsuite_b200 as W

    b, s, h = 16, 290, 32
    inp = O.make_inputs(b=b, s=s, h=h, p=64, n=64, g=1, dtype=torch.float16, seed=76)
    B, C = inp["B"].abs(), inp["C"].abs()      # (no cancellation in C.B)
    at = [32 * k + resets + 1 for k in range(s // 32)]
    X = torch.zeros_like(inp["X"])
    X[:, at] = inp["X"][:, at]
    A = torch.full_like(inp["A"], -0.01) * (1 + torch.rand(s, generator=torch.Generator().manual_seed(77)))[:, None]
    for k in range(s // 32):
        A[:, 32 * k:32 * k + resets] = decay
    Y = W.ssd_forward(X.to(DEV), A.to(DEV), B.to(DEV), C.to(DEV), 1).cpu().double()
    Yr = O.ssd_recurrence(X, A, B, C)
    rows = [l for t in at for l in range(t, (t // 32 + 1) * 32)]
    normal = Yr.abs() > 2 ** -14
    off = torch.where(normal, (Y - Yr.half().double()) / Yr, 0).sum(dim=(0, 2, 3)) / normal.sum(dim=(0, 2, 3))
    assert off[rows].abs().max().item() < 1.6e-6


@pytest.mark.parametrize("shape", [dict(b=50, s=300, h=7, g=1, n=128), dict(b=1, s=1500, h=3, g=1, n=64),
                                   dict(b=40, s=513, h=8, g=2, n=64), dict(b=1, s=4500, h=2, g=1, n=128, decay_scale=0.002),
                                   dict(b=19, s=500, h=8, g=1, n=64), dict(b=49, s=300, h=6, g=1, n=64)],
                         ids=["chained_odd", "lookback_odd", "chained_n64", "lookback_36_pieces", "lookback_76_pairs", "lookback_147_pairs"])
def test_cut_sequences_of_no_round_length(shape):
    """Sequences dealt out over the CTAs (handed on, or folded from what the CTAs before published) whose last tile is
    ragged; 50 x 7 heads are 200 pairs of which every fourth is half empty; 36 pieces are more than a warp asks for at once."""
    inp = O.make_inputs(**{"p": 64, "dtype": torch.float16, "init": True, "seed": 70, "decay_scale": 0.02, **shape})
    _check(inp, "tcgen05", 2e-2, nsegments=2)
    gen = torch.Generator().manual_seed(71)
    z = torch.randn(shape["b"], shape["s"], shape["h"], 64, generator=gen).half()
    _check(inp, "tcgen05", 2e-2, nsegments=2, z=z)


@pytest.mark.parametrize("ragged", [0, 1], ids=["tiles", "ragged"])
@pytest.mark.parametrize("b,h,n", [(1, 16, 128), (2, 6, 64), (1, 3, 128)])
@pytest.mark.parametrize("decay", ["fast", "middle", "slow", "one_slow_head", "reset", "impulse"])
def test_long_pieces_of_cut_sequences_are_scanned_once(decay, b, h, n, ragged):
    """Pieces of 44 tiles, whose decays leave nothing of the state that enters them after 2, after some 20 or after none of their
    tiles, against the same sequences uncut: the state entering a piece is a sum in another order (2^-24), of which 16-bit operands and
    results may round the other way (a few of 2^-8, in a norm 1e-3 at most)."""
    import workloadsuite_b200 as W

    tiles, (X, A, B, C), init = _long_pieces(b, h, n, ragged, decay)
    s = X.shape[1]
    if decay == "one_slow_head":
        A[:, :, h - 1] *= 1e-3
    elif decay == "reset":
        A[:, 5000::9001] = -float("inf")
    elif decay == "impulse":           # only what entered earlier is left of most pieces
        X[:, 1000:-1000] = 0.0
    kw = dict(initial_states=init, return_final_state=True, return_logdecay=True)
    whole = W.ssd_forward(X, A, B, C, 1, kernel=None if ragged else "tcgen05", nsegments=1, **kw)
    got = W.ssd_forward(X, A, B, C, 1, **kw)
    assert W.plan(X, A, B, C, 1)["nsegments"] > 1
    assert torch.allclose(got[2], whole[2], rtol=1e-6 * tiles / 32, atol=0)
    for a, c in zip(got[:2], whole[:2]):
        _same_but_for_the_order(a, c, s)
        if decay == "impulse" and a.shape[1] == s:   # element by element, far below the rest
            a, c = a.double(), c.double()
            small = (c.abs() < 1e-6 * c.abs().max()) & (c.abs() > 1e-25 * c.abs().max())
            assert small.any() and ((a - c).abs()[small] / c.abs()[small]).median().item() < 2 ** -6


def _long_pieces(b, h, n, ragged, decay, dtype=torch.bfloat16):
    """Sequences that are cut into one piece of 44 tiles a CTA; their length in tiles, X, A, B, C, and a state to start from."""
    units = b * h if ragged else b * ((h + 1) // 2)
    tiles = 44 * (148 // units)
    s = tiles * 128 + 13 * ragged
    gen = torch.Generator(DEV).manual_seed(tiles + n)
    rand = lambda *z: torch.randn(*z, generator=gen, device=DEV)
    X, B, C = rand(b, s, h, 64).to(dtype), rand(b, s, 1, n).to(dtype), rand(b, s, 1, n).to(dtype)
    rate = {"fast": 0.8, "middle": 0.06, "slow": 1e-3, "one_slow_head": 0.3, "reset": 1e-3, "impulse": 2e-3}[decay]
    init = rand(b, h, n, 64)
    return tiles, (X, -rate * torch.rand(b, s, h, generator=gen, device=DEV) * 2.0, B, C), init


def _same_but_for_the_order(a, c, s):
    """Y or final states of a cut sequence and of the same one uncut, in the norm of each head."""
    a, c = a.double(), c.double()
    assert torch.isfinite(a).all()
    dims = (1, 3) if a.shape[1] == s else (2, 3)
    assert ((a - c).square().sum(dims) / c.square().sum(dims).clamp_min(1e-60)).sqrt().max().item() < 1e-3


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("decay", ["fast", "middle"])
@pytest.mark.parametrize("n,with_init,with_dt,gate", [(128, True, True, "Dz"), (64, False, True, "z"), (128, False, False, "D"), (64, True, False, "Dz"),
                                                      (128, False, True, "")])
def test_long_pieces_with_steps_skip_and_gate(n, with_init, with_dt, gate, decay, dtype):
    """The same with everything else that a call may have; the gate is a factor behind equal sums, so the bound stays."""
    import workloadsuite_b200 as W

    tiles, (X, A, B, C), init = _long_pieces(1, 16, n, 0, decay, dtype)
    s, gen = X.shape[1], torch.Generator(DEV).manual_seed(n)
    kw = dict(initial_states=init if with_init else None, return_final_state=True)
    if with_dt:
        kw["dt"] = (0.2 + torch.rand(1, s, 16, generator=gen, device=DEV)).to(dtype)
    if "D" in gate:
        kw["D"] = torch.randn(16, generator=gen, device=DEV).to(dtype)
    if "z" in gate:
        kw["z"] = torch.randn(1, s, 16, 64, generator=gen, device=DEV).to(dtype)
    whole = W.ssd_forward(X, A, B, C, 1, nsegments=1, **kw)
    for a, c in zip(W.ssd_forward(X, A, B, C, 1, **kw), whole):
        _same_but_for_the_order(a, c, s)
    Y = W.ssd_forward(X, A, B, C, 1, **kw, out=X)[0]     # (over an input: every tile is read once more before it is written)
    assert Y.data_ptr() == X.data_ptr()
    _same_but_for_the_order(Y, whole[0], s)


@pytest.mark.parametrize("n", [64, 128])
@pytest.mark.parametrize("gate", [False, True], ids=["plain", "gate"])
@pytest.mark.parametrize("ragged", [0, 1], ids=["tiles", "ragged"])
@pytest.mark.parametrize("what", ["nan_decay", "nan_decay_first", "nan_x", "inf_init", "huge_init"])
def test_long_pieces_pass_on_what_does_not_vanish(what, ragged, gate, n):
    """A number that is not finite where the decays leave nothing of an ordinary one, in one column of a head (a decay: in the whole head), and a
    finite one that they leave something of: as far as uncut, to the end of the next piece at least.  What the calls of odd length have of
    that is done again by the recurrence, uncut or not."""
    import workloadsuite_b200 as W

    tiles, (X, A, B, C), init = _long_pieces(1, 16, n, ragged, "fast")
    s, piece = X.shape[1], 44 * 128
    upto = s + 1
    if what.startswith("nan_decay"):
        A[:, s // 2 if what == "nan_decay" else 3000, 2] = float("nan")
        init = init if what == "nan_decay" else None
    elif what == "nan_x":
        X[:, s // 2, 2, 5] = float("nan")
        upto = s + 1 if ragged else (s // 2 // piece + 2) * piece
    elif what == "inf_init":
        init[:, 2, :, 5] = float("inf")
        upto = s + 1 if ragged else piece
    else:
        A.fill_(-0.4)                  # 51.2 a tile
        X[:, :, 2, 5] = 0.0
        init[:, 2, :, 5] = 1e36
    more = {}
    if gate:
        gen = torch.Generator(DEV).manual_seed(n)
        more = {"z": 1.0 + torch.rand(X.shape, generator=gen, device=DEV).bfloat16()}
    kw = dict(initial_states=init, return_final_state=True, return_logdecay=True, **more)
    whole = W.ssd_forward(X, A, B, C, 1, nsegments=1, **kw)
    state = None if init is None else init.clone()
    in_place = {} if state is None else {"out_final_state": state}
    for got in (W.ssd_forward(X, A, B, C, 1, **kw), W.ssd_forward(X, A, B, C, 1, **{**kw, "initial_states": state}, **in_place)):
        assert torch.equal(got[2].isnan(), whole[2].isnan())
        Y, Yw = got[0][:, :upto], whole[0][:, :upto]
        assert torch.equal(Y.isfinite(), Yw.isfinite())
        if upto > s:
            assert torch.equal(got[1].isfinite(), whole[1].isfinite())
        if what == "huge_init":
            a, c = Y[0, :piece, 2, 5].double(), Yw[0, :piece, 2, 5].double()
            small = (c.abs() < 1e-33) & (c.abs() > 1e-37)     # behind e^-160
            assert small[384:].any() and ((a - c).abs()[small] / c.abs()[small]).median().item() < 2 ** -6
        else:
            assert not Yw.isfinite().all()
        keep = Yw.isfinite().all(dim=3, keepdim=True).expand_as(Yw) & (torch.arange(16, device=DEV) != 2)[:, None]
        _same_but_for_the_order(Y.where(keep, 0.0), Yw.where(keep, 0.0), Y.shape[1])


@pytest.mark.parametrize("gate", [False, True], ids=["plain", "gate"])
@pytest.mark.parametrize("b,h,n,tiles", [(1, 16, 128, 792), (2, 6, 64, 1056), (1, 16, 128, 90), (25, 4, 128, 16), (1, 3, 128, 300)],
                         ids=["long", "long_n64", "short_pieces", "two_sequences_a_cta", "odd_heads"])
def test_cut_sequences_carry_their_state_in_place(b, h, n, tiles, gate):
    """The final states over the initial ones: the same numbers, bit by bit, as in tensors of their own.  Pieces whose beginnings have different
    lengths are through with their first pass at different times, the last one ahead of the first or behind it."""
    import workloadsuite_b200 as W

    s = tiles * 128
    gen = torch.Generator(DEV).manual_seed(tiles + n)
    rand = lambda *z: torch.randn(*z, generator=gen, device=DEV)
    X, B, C, init = rand(b, s, h, 64).bfloat16(), rand(b, s, 1, n).bfloat16(), rand(b, s, 1, n).bfloat16(), 100 * rand(b, h, n, 64)
    more = {"D": rand(h).bfloat16(), "z": rand(b, s, h, 64).bfloat16()} if gate else {}
    ramp = torch.linspace(0, 1, s, device=DEV)[None, :, None]
    for start, end in ((0.5, 0.06), (0.06, 0.5), (0.06, 0.06)):
        A = -2.0 * (start + (end - start) * ramp) * torch.rand(b, s, h, generator=gen, device=DEV)
        args = (X, A, B, C, 1)
        Y, H = W.ssd_forward(*args, initial_states=init, return_final_state=True, nsegments=2, **more)
        for _ in range(3):
            state = init.clone()
            Y2, H2 = W.ssd_forward(*args, initial_states=state, return_final_state=True, out_final_state=state, nsegments=2, **more)
            assert H2.data_ptr() == state.data_ptr() and torch.equal(Y, Y2) and torch.equal(H, state)


def test_long_pieces_are_what_is_scanned_once():
    """That the sequences of the tests around this one take that way, unless their decays are slow or an output lies on an input: the piece behind
    one whose state is not finite, and no other, has its bit in the scratch set (behind the ready flags) and was walked again."""
    import ctypes

    import workloadsuite_b200 as W
    from workloadsuite_b200 import _lib, ssd

    for decay, over_x in (("fast", False), ("middle", False), ("slow", False), ("fast", True)):
        tiles, (X, A, B, C), init = _long_pieces(1, 16, 128, 0, decay)
        X[:, X.shape[1] // 2, 2, 5] = float("nan")
        args, Y = _lib.SsdArgs(), X if over_x else torch.empty_like(X)
        ssd._fill(args, X, A, B, C, None, init, Y, None, None, 1, None, None, False)
        ws = torch.zeros(_lib.load().ssd_b200_workspace_bytes(ctypes.byref(args)), dtype=torch.uint8, device=DEV)
        args.workspace, args.workspace_bytes = ws.data_ptr(), ws.numel()
        assert _lib.load().ssd_b200_forward(ctypes.byref(args), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        words = ws[296 * 128 * 64 * 4 + 1280 :].view(torch.int32)[296:301].tolist()
        cta = tiles // 44 + tiles // 2 // 44 + 1             # of the second pair of heads
        assert words == [(1 << cta % 32) * (cta // 32 == i and decay != "slow" and not over_x) for i in range(5)]


@pytest.mark.parametrize("in_place", [False, True], ids=["by_beginnings", "state_in_place"])
def test_a_lost_piece_of_a_long_sequence_is_reported(in_place):
    """The first CTA leaves without publishing: those behind it give up after 3 ms, the launch that walks pieces again has nothing to do (what they
    folded is no state), and the next forward is as ever."""
    import time

    import workloadsuite_b200 as W

    tiles, (X, A, B, C), init = _long_pieces(1, 16, 128, 0, "fast")
    run = lambda state, **kw: W.ssd_forward(X, A, B, C, 1, initial_states=state, return_final_state=True, out_final_state=state if in_place else None, **kw)
    Y, H = run(init.clone())
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    run(init.clone(), wait_limit_ms=3, inject_lost_handover=True)
    torch.cuda.synchronize()
    assert time.perf_counter() - t0 < 0.5 and W.device_status(DEV) == 6
    again = run(init.clone())
    torch.cuda.synchronize()
    assert W.device_status(DEV) == 0 and torch.equal(Y, again[0]) and torch.equal(H, again[1])


@pytest.mark.parametrize("s", [3, 8, 37, 130])
@pytest.mark.parametrize("p,n", [(64, 16), (64, 128), (32, 32), (128, 64)])
def test_fp32_scan_tokens_in_line_and_the_rest(s, p, n):
    """Steps of up to 128 tokens, several tokens in line and the remainder one by one, full and partly used states."""
    inp = O.make_inputs(b=2, s=s, h=2, p=p, n=n, g=1, dtype=torch.float32, init=True, seed=80 + s, decay_scale=0.3)
    _check(inp, "scan_f32", 1e-4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("units,s", [(8, 3), (8, 11), (304, 3), (304, 11), (304, 21), (640, 21)])
@pytest.mark.parametrize("n", [32, 64, 128])
def test_fp32_scan_with_registers_for_more_ctas(n, units, s, dtype):
    """Tokens in line or one after the other, registers for two to five CTAs of an SM: chosen by the sequences and their tokens."""
    inp = O.make_inputs(b=units // 8, s=s, h=8, p=64, n=n, g=2, dtype=dtype, init=True, seed=83 + s, decay_scale=0.3)
    _check(inp, "scan_f32", 1e-4 if dtype == torch.float32 else 2e-2, nsegments=1)


@pytest.mark.parametrize("n", [16, 32, 64, 128])
@pytest.mark.parametrize("cut", [70, 77, 123])
def test_fp32_recurrence_by_name(cut, n):
    """Token by token whatever the length: a sequence in two parts leaves the same state, bit by bit, as at once (Y's sums over the state
    may be taken in another order)."""
    import workloadsuite_b200 as W

    inp = O.make_inputs(b=2, s=200, h=4, p=64, n=n, g=2, dtype=torch.float32, init=True, seed=n, decay_scale=0.1)
    X, A, B, C, init = (inp[k].to(DEV) for k in ("X", "A", "B", "C", "initial_states"))
    run = lambda lo, hi, H: W.ssd_forward(X[:, lo:hi], A[:, lo:hi], B[:, lo:hi], C[:, lo:hi], 1, initial_states=H, return_final_state=True,
                                          kernel="scan_f32", nsegments=1)
    Y, H = run(0, 200, init)
    Y1, H1 = run(0, cut, init)
    Y2, H2 = run(cut, 200, H1)
    assert torch.equal(H, H2)
    assert (Y - torch.cat([Y1, Y2], 1)).abs().max().item() < 2 ** -20 * Y.abs().max().item()


@pytest.mark.parametrize("n", [16, 32, 64, 128])
@pytest.mark.parametrize("s", [64, 65, 79, 128, 129, 200])
@pytest.mark.parametrize("decays", ["mild", "both_signs", "resets", "strong", "growth", "x_nan", "b_inf", "huge"])
def test_fp32_tokens_side_by_side(decays, s, n):
    """Pieces of 16 tokens and tiles of 64 or 128, whole and not, and what sends a tile back to the recurrence: decays that leave the
    range of a piece, numbers that are not finite or overflow when they are scaled.  A sum of at most 144 products in fp32,
    2^-24 each, and decays known to as much: some 2e-6 of the largest term, which a result may be a few times smaller than."""
    import workloadsuite_b200 as W

    inp = O.make_inputs(b=2, s=s, h=4, p=64, n=n, g=2, dtype=torch.float32, init=True, seed=s + n, decay_scale=0.1)
    gen = torch.Generator().manual_seed(s)
    dt = 0.2 + torch.rand(2, s, 4, generator=gen)
    X, A, B, C, init = (inp[k] for k in ("X", "A", "B", "C", "initial_states"))
    at = s - 17                        # in the last but one piece, or the one before
    if decays == "both_signs":
        A = torch.randn(A.shape, generator=gen)
    elif decays == "resets":
        A[:, ::23] = -float("inf")
    elif decays == "strong":
        A = A - 20.0
    elif decays == "growth":           # 40 e-folds within a piece, gone again at once; x of nought before
        X[:, : at + 3] = 0.0
        init.zero_()
        A[:, at] = 90.0 - 50.0
        A[:, at + 2] = -40.0
    elif decays == "x_nan":
        X[:, at, 1] = float("nan")
    elif decays == "b_inf":
        B[:, at, 0] = float("inf")
    elif decays == "huge":             # finite results near the top of the range, from a tile whose decays reach e^-35
        A = torch.full_like(A, -2.2)
        X, init = X * 1e30, init * 1e30
    want, Hw = O.ssd_recurrence(X, A, B, C, dt=dt, initial_states=init, return_final_state=True)
    d = [t.to(DEV) for t in (X, A, B, C, dt, init)]
    Y, H = W.ssd_forward(d[0], d[1], d[2], d[3], 1, dt=d[4], initial_states=d[5], return_final_state=True)
    for got, ref in ((Y.cpu().double(), want), (H.cpu().double(), Hw)):
        assert torch.equal(got.isfinite(), ref.isfinite())
        ok = ref.isfinite()
        err, size = ((got - ref).where(ok, 0.0).abs(), ref.where(ok, 0.0).abs())
        dims = (1, 3) if got.dim() == 4 and got.shape[1] == s else (2, 3)
        assert (err.amax(dim=dims) / size.amax(dim=dims).clamp_min(1e-30)).max().item() < 1e-5
    Yc, Hc = W.ssd_forward(d[0], d[1], d[2], d[3], 1, dt=d[4], initial_states=d[5], return_final_state=True, nsegments=2)
    ok = Y.isfinite()
    assert torch.equal(ok, Yc.isfinite())
    if decays in ("mild", "both_signs", "strong", "resets"):
        assert (Yc - Y).abs().max().item() <= 2e-5 * Y.abs().max().item() and (Hc - H).abs().max().item() <= 2e-5 * H.abs().max().item()
    again = W.ssd_forward(d[0], d[1], d[2], d[3], 1, dt=d[4], initial_states=d[5], out=d[0])
    assert torch.equal(again.nan_to_num(), Y.nan_to_num())       # (Y over X)


@pytest.mark.parametrize("n", [16, 32, 64, 128])
@pytest.mark.parametrize("s", [64, 77, 200])
@pytest.mark.parametrize("decays", ["even", "spikes", "resets", "up_and_down"])
def test_fp32_strong_decays_keep_their_bits(decays, s, n):
    """What is left behind decays that leave the range of a piece's scaling, element by element: x in every eleventh token only, so that most of Y is
    nothing else.  Measured by the same sums of magnitudes, an element is off by the rounding of its weight (a decay e^-80 known to 2^-24 of its
    exponent: 5e-6) and of a sum of up to 128 products (128 * 2^-24 = 8e-6 at most); and by no more than the recurrence is."""
    import workloadsuite_b200 as W

    inp = O.make_inputs(b=2, s=s, h=4, p=64, n=n, g=2, dtype=torch.float32, init=True, seed=s + n, decay_scale=0.1)
    gen = torch.Generator().manual_seed(s)
    dt = 0.2 + torch.rand(2, s, 4, generator=gen)
    X, A, B, C, init = (inp[k] for k in ("X", "A", "B", "C", "initial_states"))
    X[:, torch.arange(s) % 11 != 3] = 0.0
    if decays == "even":
        A = -2.6 - torch.rand(A.shape, generator=gen)
    elif decays == "spikes":
        A[:, 5::13] = -41.0
    elif decays == "resets":
        A[:, 9::16], A[:, 40:42], A[:, 15] = -float("inf"), -float("inf"), -200.0
    elif decays == "up_and_down":
        A[:, 2::8], A[:, 4::8] = 30.0, -30.0
    want, Hw = O.ssd_recurrence(X, A, B, C, dt=dt, initial_states=init, return_final_state=True)
    size, Hs = O.ssd_recurrence(X.abs(), A, B.abs(), C.abs(), dt=dt, initial_states=init.abs(), return_final_state=True)
    d = [t.to(DEV) for t in (X, A, B, C)]
    kw = dict(dt=dt.to(DEV), initial_states=init.to(DEV), return_final_state=True)
    errors = []
    for kernel in (None, "scan_f32"):
        Y, H = W.ssd_forward(*d, 1, kernel=kernel, **kw)
        for got, ref, terms in ((Y.cpu().double(), want, size), (H.cpu().double(), Hw, Hs)):
            assert (got[terms == 0] == 0).all()
            err = ((got - ref).abs() / terms)[terms > 1e-34]        # (below, fp32 has fewer bits)
            errors += [err.square().mean().sqrt().item(), err.max().item()] if err.numel() else [0.0, 0.0]
    assert max(errors) < 1.3e-5 and errors[0] < max(1.5 * errors[4], 1e-7) and errors[2] < max(1.5 * errors[6], 1e-7), errors


@pytest.mark.parametrize("b,h,n,g", [(3, 6, 128, 2), (1, 4, 256, 1), (40, 6, 16, 3), (40, 6, 32, 2), (40, 6, 256, 6), (2, 1, 64, 1)])
def test_step_reads_strided_operands_and_d_in_its_own_type(b, h, n, g):
    """Columns of a projection's output against the same values copied out: the same arithmetic, so the same bits.  CTAs of half
    and of all columns."""
    import workloadsuite_b200 as W

    gen = torch.Generator(DEV).manual_seed(90)
    proj = torch.randn(b, 2 * h * 64 + 2 * g * n + h + 5, generator=gen, device=DEV).half()
    x, z, B, C, dt, _ = torch.split(proj, [h * 64, h * 64, g * n, g * n, h, 5], dim=-1)
    x, z, B, C = x.unflatten(-1, (h, 64)), z.unflatten(-1, (h, 64)), B.unflatten(-1, (g, n)), C.unflatten(-1, (g, n))
    a = -torch.rand(b, 2 * h, generator=gen, device=DEV)[:, ::2]
    D = torch.randn(h, generator=gen, device=DEV).half()
    S1 = torch.randn(b, h, n, 64, generator=gen, device=DEV)
    S2 = S1.clone()
    y1 = W.ssd_step(x, a, B, C, S1, dt=dt, D=D, z=z)
    y2 = W.ssd_step(x.contiguous(), a.contiguous(), B.contiguous(), C.contiguous(), S2, dt=dt.contiguous(), D=D.float(),
                    z=z.contiguous())
    assert torch.equal(y1, y2) and torch.equal(S1, S2)


def test_a_step_after_a_call_that_failed_is_made_once():
    """A call that ran out of memory leaves a CUDA error behind; the step after it, which updates the state in place, must not
    take that for its own and be made again."""
    import ctypes

    import workloadsuite_b200 as W
    from workloadsuite_b200 import _lib

    b, h, n = 2, 4, 64
    gen = torch.Generator(DEV).manual_seed(92)
    x, B, C = (torch.randn(b, k, 64, generator=gen, device=DEV).bfloat16() for k in (h, 1, 1))
    a = -torch.rand(b, h, generator=gen, device=DEV)
    S = torch.randn(b, h, n, 64, generator=gen, device=DEV)
    once, state = S.clone(), S.clone()
    y = W.ssd_step(x, a, B, C, once)
    ctx, handle = ctypes.c_void_p(), (ctypes.c_ubyte * _lib.XCHG_HANDLE_BYTES)()
    assert _lib.load().ssd_b200_xchg_create(1 << 44, 2, ctypes.byref(ctx), handle) == -6     # 32 TiB
    assert torch.equal(W.ssd_step(x, a, B, C, state), y) and torch.equal(state, once)


def test_what_pytorch_throws_in_the_binding_is_raised():
    """Tensors without sizes, allocations that cannot be made, an output that is refused: Python exceptions, of PyTorch's own
    kinds."""
    import workloadsuite_b200 as W

    nested = torch.nested.nested_tensor([torch.ones(4, 64), torch.ones(3, 64)], device=DEV)
    B, a, S = torch.ones(2, 1, 64, device=DEV), -torch.ones(2, 4, device=DEV), torch.zeros(2, 4, 64, 64, device=DEV)
    with pytest.raises(RuntimeError):
        W.ssd_step(nested, a, B, B, S)
    with pytest.raises(RuntimeError):
        W.conv1d_silu(nested, torch.ones(64, 1, 4, device=DEV))
    with pytest.raises(RuntimeError):
        W.dt_prologue(nested, None, torch.zeros(64, device=DEV))
    X = torch.ones(1, 128, 4, 64, device=DEV).bfloat16()
    A, G = -torch.ones(1, 128, 4, device=DEV), torch.ones(1, 128, 1, 64, device=DEV).bfloat16()
    with pytest.raises(RuntimeError):
        W.ssd_forward(torch.nested.nested_tensor([torch.ones(128, 4, 64), torch.ones(64, 4, 64)], device=DEV), A, G, G, 64)
    with pytest.raises(torch.OutOfMemoryError):
        W.dt_prologue(torch.zeros(1, 1, 64, device=DEV).expand(1 << 20, 1 << 20, 64), None, torch.zeros(64, device=DEV))
    with pytest.raises(ValueError, match="out_logdecay"):
        W.ssd_forward(X, A, G, G, 128, out_logdecay=torch.zeros(1, 5, device=DEV))


@pytest.mark.parametrize("dtype,l,d", [(torch.float16, 1, 64), (torch.float16, 9, 128), (torch.bfloat16, 65, 64),
                                       (torch.float32, 5, 64), (torch.float32, 67, 192), (torch.bfloat16, 2050, 4096),
                                       (torch.float16, 1780, 1024), (torch.bfloat16, 1188, 1024), (torch.float16, 1780, 3072), (torch.bfloat16, 1965, 3072), (torch.float16, 1410, 5120)])
@pytest.mark.parametrize("taps", [2, 3, 4])
def test_conv_run_lengths(dtype, l, d, taps):
    """From a run shorter than a piece to the longest run (64 tokens; the last cases 16 to 56), against the operator in fp64 (one rounding of the result, and
    tanh.approx for 16-bit types: 2^-8 of the largest value bounds both)."""
    import workloadsuite_b200 as W

    gen = torch.Generator().manual_seed(l)
    x = torch.randn(2, l, d, generator=gen).to(dtype)
    w, bias = (torch.randn(d, 1, taps, generator=gen) * 0.5).to(dtype), torch.randn(d, generator=gen).to(dtype)
    y = W.conv1d_silu(x.to(DEV), w.to(DEV), bias.to(DEV)).cpu().double()
    c = torch.nn.functional.conv1d(x.double().transpose(1, 2), w.double(), bias.double(), padding=taps - 1, groups=d)[..., :l]
    ref = torch.nn.functional.silu(c).transpose(1, 2)
    assert ((y - ref).abs().max() / ref.abs().max()).item() < (1e-5 if dtype == torch.float32 else 2 ** -8)


@pytest.mark.parametrize("dtype,l", [(torch.float16, 64), (torch.bfloat16, 33), (torch.float32, 32)])
def test_conv_in_place_up_to_the_longest_run(dtype, l):
    """A column of up to 64 tokens (fp32: 32) is one thread's, so a call that writes over its input has the bits of one that does
    not; many calls, since a race need not show in one."""
    import workloadsuite_b200 as W

    gen = torch.Generator(DEV).manual_seed(l)
    x = torch.randn(1, l, 2048, generator=gen, device=DEV).to(dtype)
    w, bias = torch.randn(2048, 1, 4, generator=gen, device=DEV).to(dtype), torch.randn(2048, generator=gen, device=DEV).to(dtype)
    want = W.conv1d_silu(x, w, bias)
    for _ in range(100):
        y = x.clone()
        W.conv1d_silu(y, w, bias, out=y)
        assert torch.equal(y, want)


def test_dt_prologue_eight_heads_per_thread():
    """More than 2^17 elements take the vector path; the functions are those of the scalar one, so its rows have the same
    bits as the first rows computed alone."""
    import workloadsuite_b200 as W

    gen = torch.Generator(DEV).manual_seed(91)
    raw = (torch.randn(4, 1031, 40 + 8, generator=gen, device=DEV) * 3 - 2).half()[..., 8:]
    bias, A_log = torch.randn(40, generator=gen, device=DEV).half(), torch.rand(40, generator=gen, device=DEV)
    dt, A = W.dt_prologue(raw, bias, A_log)
    dt1, A1 = W.dt_prologue(raw[:, :7], bias, A_log)
    assert torch.equal(dt[:, :7], dt1) and torch.equal(A[:, :7], A1)
    ref = torch.nn.functional.softplus((raw + bias).double())
    assert ((dt.double() - ref).abs() <= 2 ** -10 * ref + 2 ** -24).all()     # half an ulp, or of the smallest step


@pytest.mark.parametrize("rows", [2 ** 31 - 1024, 2 ** 31 + 1024], ids=["last_pass_past_31_bits", "rows_past_31_bits"])
def test_dt_prologue_row_counter(rows):
    """More rows than a 32-bit counter can walk (one head, the same raw value in each: 13 GB of results)."""
    import workloadsuite_b200 as W

    raw = torch.full((1, 1, 1), -1.5, device=DEV).half().expand(2, rows // 2, 1)
    A_log = torch.full((1,), 0.5, device=DEV)
    dt, A = W.dt_prologue(raw, None, A_log)
    dt1, A1 = W.dt_prologue(raw[:1, :1], None, A_log)
    assert bool((dt == dt1).all()) and bool((A == A1).all())
    del dt, A
    torch.cuda.empty_cache()


@pytest.mark.parametrize("b,s,h,n", [(3, 2048, 24, 128), (11, 384, 8, 64), (35, 512, 32, 64), (2, 4096, 80, 128)],
                         ids=["ramps_in_an_entry", "groups", "groups_of_a_large_whole", "ramps_in_an_entry_of_a_large_whole"])
def test_host_pipeline_chunks_and_sets(b, s, h, n):
    """Chunks, ramps and sets of batch entries against the device forward over the same tensors (other cuts of the
    sequence, so other roundings of the carried state's copy)."""
    import workloadsuite_b200 as W

    inp = O.make_inputs(b=b, s=s, h=h, p=64, n=n, g=1, dtype=torch.bfloat16, init=True, seed=95, decay_scale=0.05)
    d = {k: v.to(DEV) for k, v in inp.items()}
    Y, H = W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 128, initial_states=d["initial_states"], return_final_state=True)
    r = W.HostRunner(b, s, h, 64, n, 1, 128, torch.bfloat16, device=DEV)
    out, fin = torch.empty_like(inp["X"]), torch.empty(b, h, n, 64)
    r.run(inp["X"], inp["A"], inp["B"], inp["C"], out, initial_states=inp["initial_states"], final_state=fin)
    assert max(O.error_metrics(out, Y.cpu())) < 2e-2 and max(O.error_metrics(fin, H.cpu())) < 2e-2


@pytest.mark.parametrize("dtype,eps", [(torch.bfloat16, 2 ** -8), (torch.float16, 2 ** -11)])
@pytest.mark.parametrize("b,s,h,g,n,nsegments", [(2, 33, 3, 1, 128, 1), (2, 127, 4, 2, 64, 1), (1, 129, 4, 1, 128, 1), (3, 500, 4, 4, 64, 1),
                                                 (50, 300, 6, 2, 128, None), (1, 3001, 5, 1, 64, None), (1, 4700, 2, 1, 128, None)],
                         ids=["one_tile", "tile_less_one", "tile_plus_one", "whole", "chained", "lookback", "lookback_37_tiles"])
def test_fp32_scan_on_the_tensor_cores(b, s, h, g, n, nsegments, dtype, eps):
    """Products of 16-bit pieces that hold fp32 numbers: Y is off by its own rounding (eps of the value at most) and the fp32
    sums' 1e-5, as with the recurrence; the state, a sum over the tokens that decay leaves (tens), by four units of 2^-24.
    Columns of a wider tensor, as a projection's output has them, and every output of the call."""
    import workloadsuite_b200 as W

    inp = O.make_inputs(b=b, s=s, h=h, p=64, n=n, g=g, dtype=dtype, init=True, seed=80 + s, decay_scale=0.1)
    inp["A"].neg_().abs_().neg_()
    dt = (0.01 + 0.2 * torch.rand(b, s, h, generator=torch.Generator().manual_seed(s))).to(dtype)
    wide = torch.cat([inp["B"].flatten(2), inp["X"].flatten(2), inp["C"].flatten(2)], dim=-1).to(DEV)
    B, X, C = torch.split(wide, [g * n, h * 64, g * n], dim=-1)
    X, B, C = X.unflatten(-1, (h, 64)), B.unflatten(-1, (g, n)), C.unflatten(-1, (g, n))
    plan = W.plan(X, inp["A"].to(DEV), B, C, 1, nsegments=nsegments)
    assert plan["kernel"] == "scan_f32" and plan["launches"] == 2
    Y, H, ld = W.ssd_forward(X, inp["A"].to(DEV), B, C, 1, dt=dt.to(DEV), initial_states=inp["initial_states"].to(DEV),
                             return_final_state=True, return_logdecay=True, nsegments=nsegments)
    Yr, Hr = O.ssd_recurrence(inp["X"], inp["A"], inp["B"], inp["C"], dt=dt, initial_states=inp["initial_states"],
                              return_final_state=True)
    assert ((Y.cpu().double() - Yr).abs() <= eps * Yr.abs() + 1e-5 * Yr.abs().max()).all()
    assert ((H.cpu().double() - Hr).norm() / Hr.norm()).item() < 4 * 2 ** -24
    total = inp["A"].double().sum(1)
    assert ((ld.cpu().double() - total).abs() <= 2 ** -24 * total.abs()).all()      # summed in 64 bits, rounded once


def _state_of_small_numbers(s, x, dt, A=None, rows=slice(None), n=128):
    """The worst relative error (2-norm) of a head's final state, fp16, X of size x in some rows, and the same of the recurrence."""
    import workloadsuite_b200 as W

    b, h = 2, 4
    inp = O.make_inputs(b=b, s=s, h=h, p=64, n=n, g=1, dtype=torch.float16, seed=85 + s, decay_scale=0.02)
    X = torch.zeros_like(inp["X"])
    X[:, rows] = (inp["X"][:, rows].float() * x).half()
    A = -inp["A"].abs() if A is None else torch.full_like(inp["A"], A)
    step = dt * (0.5 + torch.rand(b, s, h, generator=torch.Generator().manual_seed(s)))
    step = step.half()
    run = lambda **kw: W.ssd_forward(X.to(DEV), A.to(DEV), inp["B"].to(DEV), inp["C"].to(DEV), 1, dt=step.to(DEV),
                                     return_final_state=True, **kw)[1].cpu().double()
    Hr = O.ssd_recurrence(X, A, inp["B"], inp["C"], dt=step, return_final_state=True)[1]
    off = lambda H: ((H - Hr).norm(dim=(2, 3)) / Hr.norm(dim=(2, 3))).max().item()
    return off(run()), off(run(kernel="scan_f32"))


@pytest.mark.parametrize("dt", [0.5, 1e-2, 1e-3, 1e-4])
@pytest.mark.parametrize("s", [33, 129, 300])
def test_fp16_small_steps_in_a_last_tile(s, dt):
    """The steps' unit comes from the tokens that are there: the last tile's state is as close as the others'.  A sum of up to 128
    products of 22 to 23 bits in random directions, cut off in eight accumulations (up to 2^-23 each, all downwards: four units of
    2^-24 in the mean), and the tiles' sum: five units."""
    assert _state_of_small_numbers(s, 1e-3, dt)[0] < 5 * 2 ** -24


@pytest.mark.parametrize("n", [64, 128])
@pytest.mark.parametrize("s,x,dt,A,rows", [(33, 1e-5, 1e-2, None, slice(None)), (129, 1e-4, 1e-4, None, slice(None)), (300, 1e-6, 0.5, None, slice(None)),
                                           (300, 1e-6, 1e-3, None, slice(None)), (3001, 1e-5, 1e-3, None, slice(None)), (300, 1.0, 0.5, -0.4, slice(130, 160)),
                                           (300, 1000.0, 0.5, -0.4, slice(130, 160)), (300, 1000.0, 1e-4, None, slice(None))],
                         ids=["one_tile", "last_token", "smallest", "smallest_steps", "lookback", "decayed", "decayed_large", "large"])
def test_fp16_numbers_of_any_size_keep_their_bits(s, x, dt, A, rows, n):
    """Small x, small steps, and x that 96 tokens of the tile have decayed to 1e-17 of it: six units of 2^-24 (of the eight
    accumulations' cut-offs, 16 units at most and four in the mean; the worst of eight heads), and where the decay itself is most of
    the error (38 nats in a tile, summed in fp32), no more than the recurrence."""
    here, recurrence = _state_of_small_numbers(s, x, dt, A, rows, n)
    assert here < max(6 * 2 ** -24, recurrence if A else 0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("b,s,h,n", [(2, 300, 4, 128), (1, 3001, 8, 64), (50, 300, 6, 128)], ids=["whole", "lookback", "chained"])
@pytest.mark.parametrize("what", ["x_nan", "x_inf", "b_inf", "c_nan", "a_nan", "growth", "state_inf", "overflow"])
def test_what_the_tensor_cores_cannot_do_at_fp32_is_the_recurrence_s(what, b, s, h, n, dtype):
    """Numbers that are not finite (which must not reach tokens before their own), log-decays above zero, and what overflows
    in fp16 pieces: bit by bit what the recurrence gives, in the segments that it cuts long sequences of few heads into."""
    import workloadsuite_b200 as W

    inp = O.make_inputs(b=b, s=s, h=h, p=64, n=n, g=1, dtype=dtype, init=True, seed=81, decay_scale=0.1)
    X, A, B, C, init = (inp[k] for k in ("X", "A", "B", "C", "initial_states"))
    if what == "x_nan":
        X[0, 150, 1, 3] = float("nan")
    elif what == "x_inf":
        X[0, 150, 1, 3] = float("inf")
    elif what == "b_inf":
        B[0, 150, 0, 3] = -float("inf")
    elif what == "c_nan":
        C[0, 150, 0, 3] = float("nan")
    elif what == "a_nan":
        A[0, 150, 1] = float("nan")
    elif what == "growth":
        A[0, 100:130, 1] = 1.5
    elif what == "state_inf":
        init[0, 1, 5, 5] = float("inf")
    elif what == "overflow":
        if dtype == torch.bfloat16:
            pytest.skip("bf16 has the range of fp32")
        X.mul_(8000)
    d = {k: v.to(DEV) for k, v in inp.items()}
    run = lambda **kw: W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, initial_states=d["initial_states"],
                                     return_final_state=True, **kw)
    assert W.plan(d["X"], d["A"], d["B"], d["C"], 1, kernel="scan_f32")["nsegments"] == (11 if s == 3001 else 1)
    for got, want in zip(run(), run(kernel="scan_f32")):
        assert torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0)) and torch.equal(got.isnan(), want.isnan())


def _redo_args(b, s, h, n, workspace_bytes, nsegments=0):
    """Arguments of a call that the recurrence has to do again, with scratch of the given size; and its tensors."""
    import ctypes

    from workloadsuite_b200 import _lib
    from workloadsuite_b200.ssd import _fill

    d = {k: v.to(DEV) for k, v in O.make_inputs(b=b, s=s, h=h, p=64, n=n, g=1, dtype=torch.bfloat16, init=True, seed=86,
                                                decay_scale=0.1).items()}
    d["A"][0, s // 2, 0] = 0.04
    d["Y"], d["H"], d["ld"] = torch.empty_like(d["X"]), torch.empty(b, h, n, 64, device=DEV), torch.empty(b, h, device=DEV)
    d["status"] = torch.zeros(1, dtype=torch.int32, device=DEV)
    args = _lib.SsdArgs()
    _fill(args, d["X"], d["A"], d["B"], d["C"], None, d["initial_states"], d["Y"], d["H"], d["ld"], 1, None, nsegments, False)
    args.status = d["status"].data_ptr()
    lib = _lib.load()
    size = workspace_bytes(int(lib.ssd_b200_workspace_bytes(ctypes.byref(args))))
    d["ws"] = torch.full((max(size, 1),), 0xa5, dtype=torch.uint8, device=DEV)
    args.workspace, args.workspace_bytes = d["ws"].data_ptr() if size else None, size
    run = lambda: lib.ssd_b200_forward(ctypes.byref(args), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return run, d


@pytest.mark.parametrize("b,s,h,n,least", [(1, 5001, 3, 128, False), (2, 1025, 24, 64, False), (1, 700, 1, 128, False), (1, 9001, 1, 64, False),
                                           (1, 5001, 48, 128, False), (1, 5001, 48, 128, True)])
def test_a_call_that_is_done_again_is_cut_as_the_scratch_allows(b, s, h, n, least):
    """With the scratch that it asks for the recurrence cuts the sequences, with the least it does not; all outputs bit by bit, twice in
    a row on scratch that holds the first call's counters."""
    import workloadsuite_b200 as W

    run, d = _redo_args(b, s, h, n, lambda asked: 768 + 2 * 148 * n * 64 * 4 + 2 * 1280 if least else asked)
    want = W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, initial_states=d["initial_states"], return_final_state=True,
                         return_logdecay=True, kernel="scan_f32", nsegments=1 if least else None)
    for _ in range(2):
        assert run() == 0
        torch.cuda.synchronize()
        assert d["status"].item() == 0
        for got, w in zip((d["Y"], d["H"], d["ld"]), want):
            assert torch.equal(got, w)


@pytest.mark.parametrize("b,s,h,n", [(1, 20001, 24, 128), (1, 60001, 8, 64), (1, 3001, 120, 128)])
def test_a_call_that_is_done_again_takes_what_the_recurrence_takes(b, s, h, n):
    """1 x 20 001 tokens of 24 heads: 1.6 ms and some 0.3 for the kernel ahead and the joints in one launch, not the 6 ms of whole
    sequences."""
    import workloadsuite_b200 as W

    run, d = _redo_args(b, s, h, n, lambda asked: asked)
    scan = lambda: W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, initial_states=d["initial_states"], return_final_state=True,
                                 kernel="scan_f32")
    ms = []
    for f in (run, scan):
        f()
        best = 1e9
        for _ in range(5):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            f()
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        ms.append(best)
    assert ms[0] < 1.4 * ms[1]


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("b,s,h,n", [(1, 4099, 37, 128), (2, 3001, 80, 64), (1, 700, 1, 128), (2, 300, 4, 64)])
def test_scratch_asked_for_by_shape_is_enough_for_a_call_of_the_recurrence(b, s, h, n, offset):
    """A size asked for without pointers, as the sizing of a pipeline's scratch does; the state leaves where it entered, or is only
    4-byte aligned as well, which makes the call the recurrence's: in segments of its own (37 heads, one) or whole (160)."""
    import ctypes

    import workloadsuite_b200 as W
    from workloadsuite_b200 import _lib
    from workloadsuite_b200.ssd import _fill

    d = {k: v.to(DEV) for k, v in O.make_inputs(b=b, s=s, h=h, p=64, n=n, g=1, dtype=torch.bfloat16, init=True, seed=87,
                                                decay_scale=0.1).items()}
    args, lib = _lib.SsdArgs(), _lib.load()
    _fill(args, d["X"], d["A"], d["B"], d["C"], None, None, None, None, None, 1, None, 0, False)
    for name in ("X", "A", "B", "C"):
        setattr(args, name, None)
    size = int(lib.ssd_b200_workspace_bytes(ctypes.byref(args)))
    state = torch.empty(b * h * n * 64 + 4, device=DEV)[offset:offset + b * h * n * 64].view(b, h, n, 64).copy_(d["initial_states"])
    Y, ws = torch.empty_like(d["X"]), torch.empty(max(size, 1), dtype=torch.uint8, device=DEV)
    _fill(args, d["X"], d["A"], d["B"], d["C"], None, state, Y, state, None, 1, None, 0, False)
    args.workspace, args.workspace_bytes = ws.data_ptr(), size
    assert lib.ssd_b200_forward(ctypes.byref(args), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    want = W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, initial_states=d["initial_states"], return_final_state=True,
                         kernel="scan_f32", nsegments=1 if b * h > 74 else None)
    assert torch.equal(Y, want[0]) and torch.equal(state, want[1])


@pytest.mark.parametrize("b,s,h,n,nsegments", [(2, 300, 4, 64, 0), (50, 300, 6, 128, 0), (1, 3001, 8, 64, 1)])
@pytest.mark.parametrize("size", [0, 512])
def test_whole_sequences_need_no_scratch(size, b, s, h, n, nsegments):
    """Without any, or with less than the tensor-core kernel can do with: the recurrence over whole sequences, which never needed some."""
    import workloadsuite_b200 as W

    run, d = _redo_args(b, s, h, n, lambda asked: size, nsegments)
    assert run() == 0
    want = W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, initial_states=d["initial_states"], return_final_state=True,
                         return_logdecay=True, kernel="scan_f32", nsegments=1)
    for got, w in zip((d["Y"], d["H"], d["ld"]), want):
        assert torch.equal(got, w)


@pytest.mark.parametrize("again", [False, True])
@pytest.mark.parametrize("b,s,h,n", [(2, 300, 4, 64), (1, 2001, 18, 128), (40, 300, 5, 128)], ids=["whole", "cut", "too_many_to_fuse"])
def test_y_written_over_the_gates(b, s, h, n, again):
    """The gates must be read before Y replaces them, also where the call has to be done by the recurrence: the same Y as elsewhere, to
    its rounding (another kernel's sums) and that of many tiles' separate skip and gate, 2^-8 each."""
    import workloadsuite_b200 as W

    d = {k: v.to(DEV) for k, v in O.make_inputs(b=b, s=s, h=h, p=64, n=n, g=1, dtype=torch.bfloat16, init=True, seed=88,
                                                decay_scale=0.1).items()}
    if again:
        d["A"][0, 10:40, 0] = 0.04
    gen = torch.Generator(DEV).manual_seed(s)
    D, z = torch.randn(h, generator=gen, device=DEV), (3 * torch.randn(b, s, h, 64, generator=gen, device=DEV)).bfloat16()
    run = lambda z, out: W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, initial_states=d["initial_states"], D=D, z=z, out=out)
    want = run(z, torch.empty_like(z)).double()
    out = z.clone()
    assert run(out, out) is out
    assert ((out.double() - want).abs() <= 2 ** -6 * want.abs() + 2 ** -8 * want.abs().max()).all()
    assert ((out.double() - want).norm() / want.norm()).item() < 2 ** -7


def test_scratch_of_calls_on_two_streams_is_their_own():
    import workloadsuite_b200 as W

    sets = [{k: v.to(DEV) for k, v in O.make_inputs(b=2, s=3001, h=80, p=64, n=128, g=1, dtype=torch.bfloat16, seed=83 + i,
                                                    decay_scale=0.1).items()} for i in range(2)]
    run = lambda d: W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, return_final_state=True)
    want = [run(d) for d in sets]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(8):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                got[i].append(run(sets[i]))
    torch.cuda.synchronize()
    for i in range(2):
        for Y, H in got[i]:
            assert torch.equal(Y, want[i][0]) and torch.equal(H, want[i][1])


@pytest.mark.parametrize("dtype,eps", [(torch.bfloat16, 2 ** -8), (torch.float16, 2 ** -11)])
@pytest.mark.parametrize("b,s,h,g,n", [(2, 65, 4, 2, 128), (1, 300, 3, 1, 64), (1, 2001, 18, 1, 128), (40, 300, 5, 1, 128)],
                         ids=["one_tile", "three", "lookback", "too_many_to_fuse"])
@pytest.mark.parametrize("which", ["D", "z", "both", "z_rows_apart"])
def test_skip_and_gate_of_the_fp32_scan(which, b, s, h, g, n, dtype, eps):
    """(Y + x D) silu(z) in fp32 ahead of the one rounding: off by that (eps of the value at most), the sums' 1e-5 and the gate's
    (exp and a division, some 2^-21 each), against the gate's size; many tiles, which are not fused; and what the recurrence has
    to do again, with both."""
    import workloadsuite_b200 as W

    inp = O.make_inputs(b=b, s=s, h=h, p=64, n=n, g=g, dtype=dtype, init=True, seed=90 + s, decay_scale=0.1)
    gen = torch.Generator().manual_seed(s)
    D = torch.randn(h, generator=gen).to(dtype) if which in ("D", "both") else None
    z = 3 * torch.randn(b, s, h, 64, generator=gen)
    z = z.to(dtype) if which != "D" else None
    d = {k: v.to(DEV) for k, v in inp.items()}
    zd = None if z is None else z.to(DEV)
    if which == "z_rows_apart":       # columns of a wider tensor
        wide = torch.zeros(b, s, h * 64 + 24, dtype=dtype, device=DEV)
        wide[..., 8:8 + h * 64] = zd.flatten(2)
        zd = wide[..., 8:8 + h * 64].unflatten(-1, (h, 64))
    run = lambda **kw: W.ssd_forward(d["X"], d["A"], d["B"], d["C"], 1, initial_states=d["initial_states"], z=zd,
                                     D=None if D is None else D.to(DEV), **kw)
    Yr = O.ssd_recurrence(inp["X"], inp["A"], inp["B"], inp["C"], initial_states=inp["initial_states"])
    size = Yr.abs().max()
    gate = torch.ones(()) if z is None else torch.nn.functional.silu(z.double())
    if D is not None:
        Yr = Yr + inp["X"].double() * D.double()[:, None]
    Yr = Yr * gate
    got, apart = run().cpu().double(), run(separate_epilogue=True).cpu().double()
    # in a kernel of their own Y has a rounding ahead of them as well
    twice = 2.1 * eps * (Yr.abs() + size * eps) + 1e-5 * size * (1 + gate.abs()) + eps * size * gate.abs()
    assert ((apart - Yr).abs() <= twice).all()
    if b * h * ((s + 127) // 128) <= 2 * 148:
        assert ((got - Yr).abs() <= eps * Yr.abs() + (1e-5 * size + 2 ** -20 * Yr.abs()) * (1 + gate.abs())).all()
    else:                                    # more tiles than that: not in the kernel
        assert torch.equal(got, apart)
    # growth (above 1/32): done again by the recurrence, where Y has a rounding before the skip and the gate; e^1.2 in all, or
    # Y times the gate overflows fp16 in both
    d["A"][0, 10:40, 0] = 0.04
    again, want = run().double(), run(kernel="scan_f32").double()
    assert ((again - want).abs() <= 2.1 * eps * want.abs() + 2 * eps * want.abs().max()).all()
    assert torch.equal(run(separate_epilogue=True).double(), want)
