"""Newton-Schulz drivers: CPU math, and the CUDA kernels against the CPU/PyTorch oracle."""
import pytest
import torch

from dion_b200.ops import newton_schulz as NS


def _orth_err(X):
    X = X.float()
    if X.size(-2) > X.size(-1):
        X = X.mT
    eye = torch.eye(X.size(-2), device=X.device)
    return ((X @ X.mT) - eye).abs().max().item()


@pytest.mark.parametrize("name,fn", [("quintic", NS.newton_schulz_quintic),
                                     ("polar_express", NS.polar_express),
                                     ("aol", NS.newton_schulz_aol),
                                     ("gram", NS.gram_newton_schulz)])
@pytest.mark.parametrize("shape", [(48, 48), (32, 96), (96, 32), (3, 40, 64)])
def test_cpu_orthogonality(name, fn, shape):
    torch.manual_seed(0)
    G = torch.randn(*shape)
    X = fn(G)
    assert X.shape == G.shape and X.dtype == torch.bfloat16
    assert _orth_err(X) < 0.35  # five bf16 iterations leave singular values in [0.7, 1.2]


def test_classic_matches_reference_coeffs(ref_dion):
    from dion.muon_reference import zeropower_via_newtonschulz5 as ref_ns
    torch.manual_seed(0)
    G = torch.randn(64, 96)
    got = NS.newton_schulz_classic(G, epsilon=1e-7, steps=5)
    assert (got.float() - ref_ns(G, 5, 1e-7).float()).abs().max().item() < 2e-2


def test_cpu_matches_reference(ref_dion):
    from dion.muon import zeropower_via_newtonschulz5
    from dion.polar_express import polar_express
    torch.manual_seed(0)
    G = torch.randn(4, 64, 96)
    assert torch.equal(NS.newton_schulz_quintic(G, 1e-7), zeropower_via_newtonschulz5(G, 1e-7))
    assert (NS.polar_express(G, 1e-6).float() - polar_express(G, 1e-6).float()).abs().max() < 2e-2


def test_buffer_form_is_for_the_drivers_alone():
    import functools

    @functools.wraps(NS.polar_express)
    def wrapped(X, epsilon=1e-6):
        return NS.polar_express(X, epsilon)

    cuda = torch.device("cuda", 0)
    assert NS.buffer_form(NS.polar_express, (4, 64, 128), cuda)
    assert not NS.buffer_form(wrapped, (4, 64, 128), cuda)
    assert not NS.buffer_form(lambda X, epsilon=None: X, (4, 64, 128), cuda)
    assert not NS.buffer_form(NS.polar_express, (4, 64, 100), cuda)
    assert not NS.buffer_form(NS.polar_express, (4, 64, 128), torch.device("cpu"))


@pytest.fixture
def products_on_cpu(monkeypatch):
    """The CUDA drivers with their kernels replaced by plain torch, to follow their buffers."""
    from dion_b200.ops import foreach as F
    from dion_b200.ops import gemm

    def ns_gemm(A, B, out=None, a_is_km=False, b_is_kn=False, D=None, alpha=1.0, beta=0.0,
                scale=None, alpha_pow=0, beta_pow=0, sym=False, extra=None):
        A, B = A.float(), B.float()
        s = scale.view(-1, 1, 1) if scale is not None else 1.0
        r = alpha * s ** alpha_pow * ((A.mT if a_is_km else A) @ (B if b_is_kn else B.mT))
        if D is not None:
            r = r + beta * s ** beta_pow * D.float()
        r = r.to(torch.bfloat16)
        return r if out is None else out.copy_(r)

    def aol_rescale_(X, A, eps):
        s = A.float().abs().sum(-1).clamp_min(eps).rsqrt()
        X.copy_(X.float() * s.unsqueeze(-1))
        A.copy_(A.float() * s.unsqueeze(-1) * s.unsqueeze(-2))

    monkeypatch.setattr(gemm, "ns_gemm", ns_gemm)
    monkeypatch.setattr(F, "aol_rescale_", aol_rescale_)
    for name in ("persistent_fits", "iterate_in_one_call"):
        monkeypatch.setattr(gemm, name, lambda *a: False)
    monkeypatch.setattr(NS, "_norm_scale", lambda X, mult, eps, part: 1.0 / (
        X.float().square().sum(dim=(1, 2)).sqrt() * mult + eps))
    monkeypatch.setattr(NS, "_use_cuda", lambda G: True)


_DRIVERS = {"polar_express": NS.polar_express, "aol": NS.newton_schulz_aol,
            "gram": NS.gram_newton_schulz}


@pytest.mark.parametrize("pending", [False, True])
@pytest.mark.parametrize("shape", [(2, 16, 40), (2, 40, 16), (24, 24)])
@pytest.mark.parametrize("variant", list(_DRIVERS))
def test_input_is_kept_and_not_returned(products_on_cpu, variant, shape, pending):
    """Dense bf16 input is read in place: a plain tensor, and the pending result of a functional
    collective, whose own address is not that of its data."""
    from torch.distributed._functional_collectives import AsyncCollectiveTensor
    torch.manual_seed(0)
    G = torch.randn(shape).bfloat16()
    before = G.clone()
    got = _DRIVERS[variant](AsyncCollectiveTensor(G) if pending else G)
    assert torch.equal(G, before)
    assert got.untyped_storage().data_ptr() != G.untyped_storage().data_ptr()
    assert torch.equal(got, _DRIVERS[variant](before))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_lazily_negated_input_is_resolved_before_its_address_is_used(dtype, monkeypatch):
    from dion_b200.ops import foreach as F
    G = torch.randn(2, 16, 40).to(dtype)
    seen = []
    monkeypatch.setattr(F, "ns_prepare", lambda X, *a, **kw: (seen.append(X) or X, None))
    X = NS._prepare_cuda(torch._neg_view(G))[0]
    assert not X.is_neg() and torch.equal(X, -G)


@pytest.mark.parametrize("shape", [(2, 16, 40), (40, 16)])
def test_no_steps_give_a_copy(products_on_cpu, shape):
    G = torch.randn(shape).bfloat16()
    got = NS.newton_schulz_classic(G, steps=0)
    assert torch.equal(got, G)
    assert got.untyped_storage().data_ptr() != G.untyped_storage().data_ptr()


def test_one_launch_loops_in_flight_have_their_own_counters(monkeypatch):
    """A second launch issued while the first one is running (another stream or thread of the same
    device) counts its barrier elsewhere."""
    from dion_b200.ops import _backend, gemm
    seen = []

    class Lib:
        def dion_ns_persistent(self, *args):
            seen.append(args[14].value)
            if len(seen) == 1:
                launch()
            return 0

    def launch():
        X, A = torch.zeros(1, 64, 128), torch.zeros(1, 64, 64)
        gemm.ns_persistent(X, torch.zeros_like(X), A, torch.zeros_like(A), NS.QUINTIC_COEFFS, None)

    monkeypatch.setattr(_backend, "lib", lambda stem: Lib())
    monkeypatch.setattr(gemm, "sm_count", lambda dev: 148)
    monkeypatch.setattr(gemm, "status_tensor", lambda dev: torch.zeros(4, dtype=torch.int32))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream",
                        lambda dev=None: type("Stream", (), {"cuda_stream": 0})())
    launch()
    assert len(seen) == 2 and 0 not in seen and seen[0] != seen[1]


@pytest.mark.gpu
def test_one_launch_loops_on_two_streams():
    """Grids that fit the GPU together, of different sizes and phase lengths: the bits of the same
    calls one after the other."""
    from dion_b200.ops import gemm
    torch.manual_seed(0)
    Gs = [torch.randn(1, m, n, device="cuda").bfloat16()
          for m, n in ((256, 256), (384, 512), (256, 1024), (512, 384))]
    for G in Gs:
        assert gemm.persistent_fits(G, *G.shape, 5)
    alone = [NS.polar_express(G) for G in Gs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(20):
        outs = []
        for i, G in enumerate(Gs):
            with torch.cuda.stream(streams[i % 2]):
                outs.append(NS.polar_express(G))
        torch.cuda.synchronize()
        for a, b in zip(alone, outs):
            assert torch.equal(a, b)
    gemm.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("form", ["dense", "odd", "two_dims", "four_dims", "transposed", "columns",
                                  "off_by_one", "one_row"])
@pytest.mark.parametrize("variant", ["polar_express", "aol", "gram"])
def test_cuda_input_forms(variant, form, dtype):
    """The input is read in place or in one rounding / padding pass, whatever its order and
    strides, and is never written."""
    fn = {"polar_express": NS.polar_express, "aol": NS.newton_schulz_aol,
          "gram": NS.gram_newton_schulz}[variant]
    torch.manual_seed(0)
    G = {"dense": lambda: torch.randn(3, 96, 200), "odd": lambda: torch.randn(3, 101, 57),
         "two_dims": lambda: torch.randn(136, 264), "four_dims": lambda: torch.randn(2, 2, 64, 72),
         "transposed": lambda: torch.randn(3, 200, 96), "columns": lambda: torch.randn(3, 96, 300),
         "off_by_one": lambda: torch.randn(3 * 96 * 200 + 1),
         "one_row": lambda: torch.randn(2, 1, 40)}[form]().to("cuda", dtype)
    if form == "transposed":
        G = G.mT
    elif form == "columns":
        G = G[:, :, 50:250]
    elif form == "off_by_one":
        G = G[1:].view(3, 96, 200)
    before = G.clone()
    got = fn(G)
    assert torch.equal(G, before) and got.shape == G.shape and got.dtype == torch.bfloat16
    m, n = G.shape[-2:]
    dense = torch.zeros(*G.shape[:-2], -(-m // 8) * 8, -(-n // 8) * 8, device="cuda",
                        dtype=torch.bfloat16)
    dense[..., :m, :n] = G
    ref = fn(dense)[..., :m, :n]
    rel = (got.float() - ref.float()).norm() / ref.float().norm()
    # the same products on the same bf16 input; only the last bits of the input's norm may differ,
    # which moves single roundings (2^-9) of fifteen products
    assert rel.item() < 2e-2, rel.item()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, 1, 1), (5, 13, 29), (2, 64, 65), (3, 100, 96), (2, 517, 1031)])
def test_prepare_rounds_pads_and_sums(shape, dtype):
    from dion_b200.ops import foreach as F
    torch.manual_seed(0)
    G = torch.randn(*shape, device="cuda").to(dtype)
    mp, np_ = (shape[1] + 7) // 8 * 8, (shape[2] + 7) // 8 * 8
    X, ss = F.ns_prepare(G, mp, np_)
    ref = torch.zeros(shape[0], mp, np_, device="cuda", dtype=torch.bfloat16)
    ref[:, :shape[1], :shape[2]] = G
    assert torch.equal(X, ref)
    exact = ref.double().square().sum(dim=(1, 2))
    assert ((ss - exact).abs() <= 1e-5 * exact).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, 768, 768), (1, 104, 2048), (3, 517, 1031)])
def test_cuda_driver_repeats_exactly(shape, dtype):
    """The same input gives the same bits: one launch, padded, one matrix or several; the sum of
    squares over tens of blocks included."""
    from dion_b200.ops import foreach as F
    torch.manual_seed(0)
    G = (torch.randn(*shape, device="cuda") * 1e-3).to(dtype)
    first = NS.polar_express(G)
    X = G.bfloat16()
    ss = F.sumsq(X)
    assert ((ss - X.double().square().sum(dim=(1, 2))).abs() <= 1e-6 * ss).all()
    for _ in range(24):
        assert torch.equal(F.sumsq(X), ss)
        assert torch.equal(NS.polar_express(G), first)
    total = ss.clone()
    assert torch.equal(F.sumsq(X, out=total), 2 * ss)


@pytest.mark.gpu
@pytest.mark.parametrize("variant", ["quintic", "classic", "polar_express", "aol", "gram"])
@pytest.mark.parametrize("shape", [(6, 768, 768), (2, 768, 3072), (2, 3072, 768), (3, 192, 768),
                                   (1, 100, 52), (256, 256)])
def test_cuda_vs_torch(variant, shape):
    from dion_b200.ops.gemm import check_status
    fn = {"quintic": NS.newton_schulz_quintic, "classic": NS.newton_schulz_classic,
          "polar_express": NS.polar_express, "aol": NS.newton_schulz_aol,
          "gram": NS.gram_newton_schulz}[variant]
    torch.manual_seed(0)
    G = torch.randn(*shape, device="cuda")
    got = fn(G)
    torch.cuda.synchronize()
    check_status()
    ref = NS.torch_reference(variant)(G)
    assert got.shape == G.shape and got.dtype == torch.bfloat16
    # Entries of an orthogonalized matrix are O(1/sqrt(n)), so a bound on the largest absolute
    # difference says little: compare every matrix by its relative Frobenius error.  Two bf16
    # evaluations of the same five iterations differ by a few percent (different accumulation
    # order and rounding points); a wrong coefficient or operand gives errors of order one.
    # Gram-NS keeps less precision in the small matrix it iterates on.
    g3 = got.float().reshape(-1, *got.shape[-2:])
    r3 = ref.float().reshape(-1, *ref.shape[-2:])
    rel = (g3 - r3).flatten(1).norm(dim=1) / r3.flatten(1).norm(dim=1)
    assert rel.max().item() < (0.2 if variant == "gram" else 0.1), rel.tolist()
    assert _orth_err(got) < 0.4


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 768, 768), (4, 768, 768), (1, 768, 3072), (1, 3072, 768),
                                   (3, 200, 136), (1, 1024, 1024)])
def test_one_launch_loop_matches_per_gemm_launches(shape, monkeypatch):
    """Small batches run all fifteen GEMMs of the loop in one cooperative launch with grid-wide
    barriers between them; the result is that of the three-launches-per-iteration path."""
    from dion_b200.ops import _backend, gemm
    from dion_b200.ops.gemm import check_status
    torch.manual_seed(1)
    G = torch.randn(*shape, device="cuda")
    monkeypatch.setenv("DION_B200_PERSISTENT_NS", "0")
    ref = NS.newton_schulz_quintic(G)
    monkeypatch.setenv("DION_B200_PERSISTENT_NS", "1")
    assert gemm.persistent_fits(G.bfloat16().contiguous(), *shape, 5)
    before = _backend.launch_count()
    got = NS.newton_schulz_quintic(G)
    launches = _backend.launch_count() - before
    torch.cuda.synchronize()
    check_status()
    assert launches <= 3                          # norm (2 kernels) + the loop
    g3, r3 = got.float().reshape(-1, *shape[-2:]), ref.float().reshape(-1, *shape[-2:])
    rel = (g3 - r3).flatten(1).norm(dim=1) / r3.flatten(1).norm(dim=1)
    assert rel.max().item() < 2e-2, rel.tolist()
    assert _orth_err(got) < 0.4
    # Bitwise repeatable for a given input scale (the scale itself comes from floating-point
    # atomics, so whole calls are only repeatable to the last bit of the scale); also shows that
    # the barrier counter is left at zero.
    B_, m, n = shape
    g = min(m, n)
    X0 = G.bfloat16().contiguous()
    scale = (1.0 / (X0.float().flatten(1).norm(dim=1) + 1e-7)).contiguous()
    outs = []
    for _ in range(3):
        X = X0.clone()
        bufs = [torch.empty_like(X), torch.empty(B_, g, g, device="cuda", dtype=torch.bfloat16),
                torch.empty(B_, g, g, device="cuda", dtype=torch.bfloat16)]
        outs.append(gemm.ns_persistent(X, bufs[0], bufs[1], bufs[2], NS.QUINTIC_COEFFS,
                                       scale).clone())
    torch.cuda.synchronize()
    check_status()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


def _exact64(X, coeffs):
    X = X.double()
    X = X / X.flatten(1).norm(dim=1)[:, None, None]
    if X.size(1) > X.size(2):
        return _exact64(X.mT, coeffs).mT
    for a, b, c in coeffs:
        A = X @ X.mT
        X = a * X + (b * A + c * (A @ A)) @ X
    return X


@pytest.mark.gpu
@pytest.mark.parametrize("spectrum", ["gradient", "dominant", "decaying"])
@pytest.mark.parametrize("groups", [(1,), (2, 1), (2, 1, 1), (2, 2, 1), (2, 2, 1, 1)])
@pytest.mark.parametrize("shape", [(2, 512, 1032), (1, 2064, 520), (3, 768, 1536), (1, 1032, 2568)])
def test_composed_steps_are_as_close_as_plain_ones(shape, groups, spectrum):
    """The composed loop is nearer to fp64 than the plain one (0.6-0.95 of its error over such
    inputs), whatever the groups, with the input left as it is."""
    from dion_b200.ops import foreach as F
    from dion_b200.ops import gemm
    torch.manual_seed(sum(shape))
    b, m, n = shape
    X = torch.randn(shape, device="cuda")
    if spectrum == "gradient":
        X *= (0.5 * torch.randn(b, m, 1, device="cuda")).exp()
    elif spectrum == "dominant":
        u, v = torch.randn(b, m, 4, device="cuda"), torch.randn(b, 4, n, device="cuda")
        X = u @ v + X
    else:
        U, S, V = torch.linalg.svd(X, full_matrices=False)
        X = (U / (1.0 + torch.arange(S.size(1), device="cuda"))) @ V
    X = X.bfloat16()
    coeffs = (NS.POLAR_EXPRESS_COEFFS + NS.POLAR_EXPRESS_COEFFS[-1:])[:sum(groups)]
    exact = _exact64(X, coeffs)
    keep = X.clone()
    scale = F.scale_of_parts(F.sumsq_parts(X), 1.0, 0.0)
    got = gemm.ns_compose(X, torch.empty_like(X), coeffs, groups, scale, torch.empty_like(X))
    g = min(m, n)
    A = torch.empty(b, g, g, device="cuda", dtype=torch.bfloat16)
    plain = gemm.ns_iterate(X, torch.empty_like(X), A, torch.empty_like(A), coeffs, scale,
                            torch.empty_like(X))
    gemm.check_status()
    err = lambda Y: ((Y.double() - exact).norm() / exact.norm()).item()  # noqa: E731
    assert err(got) <= 1.02 * err(plain)
    assert torch.equal(X, keep)


def test_which_loops_are_composed():
    from dion_b200.ops import gemm
    assert gemm.compose_groups(64, 768, 3072, 5, 148) == (2, 2, 1)
    assert gemm.compose_groups(64, 768, 3072, 6, 148) == (2, 2, 1, 1)
    assert gemm.compose_groups(24, 8192, 2048, 4, 148) == (2, 1, 1)
    assert gemm.compose_groups(64, 768, 3072, 2, 148) is None      # no pair with a step after it
    assert gemm.compose_groups(64, 768, 768, 5, 148) is None       # as many products either way
    assert gemm.compose_groups(64, 504, 8192, 5, 148) is None      # less exact below 512
    assert gemm.compose_groups(64, 772, 3072, 5, 148) is None      # not for TMA


@pytest.mark.gpu
@pytest.mark.parametrize("resets", [(2,), (), (1, 3), (4,), (0, 2, 9)])
@pytest.mark.parametrize("shape", [(1, 768, 768), (3, 136, 264), (2, 1032, 520), (4, 8, 64)])
def test_gram_in_one_call_equals_its_products_one_by_one(shape, resets, monkeypatch):
    """The same launches in the same order, so the same bits."""
    from dion_b200.ops import gemm
    torch.manual_seed(3)
    G = torch.randn(shape, device="cuda").bfloat16()
    keep = G.clone()
    got = NS.gram_newton_schulz(G, reset_iterations=resets)
    monkeypatch.setattr(gemm, "iterate_in_one_call", lambda *a: False)
    product = gemm.ns_gemm
    monkeypatch.setattr(gemm, "ns_gemm", lambda *a, **k: product(*a, **k, pair=True))
    ref = NS.gram_newton_schulz(G, reset_iterations=resets)
    gemm.check_status()
    assert torch.equal(got, ref) and torch.equal(G, keep)
    short = NS.gram_newton_schulz(G, reset_iterations=resets, coeffs=NS.POLAR_EXPRESS_COEFFS[:1])
    monkeypatch.undo()
    assert torch.equal(short, NS.gram_newton_schulz(G, reset_iterations=resets,
                                                    coeffs=NS.POLAR_EXPRESS_COEFFS[:1]))
