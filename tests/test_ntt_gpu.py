"""GPU parity of the batched NTT / INTT against the CPU golden model, through
the C ABI. Bit-exact: every output word must match."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rand_poly(rng, primes, gidx, n, polys=None):
    shape = (n,) if polys is None else (polys, n)
    cols = [rng.integers(0, int(primes[g]), shape, dtype=np.uint64).astype(np.uint32) for g in gidx]
    return np.stack(cols, axis=0 if polys is None else 1)


def test_ntt_matches_oracle_all_primes(engine40, oracle40):
    rng = np.random.default_rng(11)
    g = np.arange(engine40.num_primes)
    a = rand_poly(rng, oracle40.primes, g, oracle40.n)
    # edge values in the first words of every limb
    for l, gi in enumerate(g):
        q = int(oracle40.primes[gi])
        a[l, :4] = [0, q - 1, 1, q - 1]
    for mc in (False, True):
        assert np.array_equal(engine40.ntt(a, g, mc), oracle40.ntt(a, g, mc))


def test_intt_matches_oracle_all_primes(engine40, oracle40):
    rng = np.random.default_rng(12)
    g = np.arange(engine40.num_primes)
    a = rand_poly(rng, oracle40.primes, g, oracle40.n)
    k = np.array([rng.integers(1, int(oracle40.primes[gi])) for gi in g], dtype=np.uint32)
    assert np.array_equal(engine40.intt(a, g), oracle40.intt(a, g))
    assert np.array_equal(engine40.intt(a, g, mont_keep=True), oracle40.intt(a, g, mont_keep=True))
    for cen in (False, True):
        assert np.array_equal(engine40.intt(a, g, k, centred=cen), oracle40.intt(a, g, k, centred=cen))


def test_config1_batch_roundtrip_and_sample_parity(engine40, oracle40):
    """Config 1: 16 polynomials x the first 40 Q limbs; forward then inverse
    is the identity at full size, and two polynomials are checked word for
    word against the golden model."""
    rng = np.random.default_rng(13)
    g = engine40.level_limbs(28)[:40]
    a = rand_poly(rng, oracle40.primes, g, oracle40.n, polys=16)
    d = engine40.to_dev(a)
    f = engine40.torch.empty_like(d)
    engine40.ntt_(f, d, g)
    back = engine40.torch.empty_like(d)
    engine40.intt_(back, f, g, mont_keep=True)
    assert np.array_equal(engine40.to_host(back), a)
    fh = engine40.to_host(f)
    for p in (0, 15):
        assert np.array_equal(fh[p], oracle40.ntt(a[p], g))
    # in place
    engine40.ntt_(d, d, g)
    assert np.array_equal(engine40.to_host(d), fh)


def test_single_limb_and_subset(engine40, oracle40):
    rng = np.random.default_rng(14)
    for g in ([58], [0, 46, 47], [5]):
        a = rand_poly(rng, oracle40.primes, g, oracle40.n)
        assert np.array_equal(engine40.ntt(a, g), oracle40.ntt(a, g))


def test_bad_arguments_fail_loudly(engine40, pkg):
    a = engine40.empty(1, engine40.n)
    with pytest.raises(pkg.CfheError):
        engine40.ntt_(a, a, [engine40.num_primes])


def view_at(e, words, polys, limbs, offset, extra):
    """A [polys, limbs, N] view `offset` words into a buffer on a 16-byte
    boundary, polynomials limbs * N + extra words apart."""
    stride = limbs * e.n + extra
    buf = e.torch.empty(offset + polys * stride, dtype=e.torch.int32, device="cuda:0")
    v = buf.as_strided((polys, limbs, e.n), (stride, e.n, 1), offset)
    v.copy_(words)
    return v


@pytest.mark.parametrize("offset,extra", [(1, 0), (2, 0), (3, 1), (0, 1), (4, 2), (0, 7)])
def test_sides_that_may_start_at_any_word(engine40, offset, extra):
    """The source of a forward and the destination of an inverse transform, off
    the 8- and 16-byte boundaries by offset or by stride."""
    e = engine40
    rng = np.random.default_rng(15)
    g = [0, 20, 50]  # an auxiliary prime above 2^30 among them
    a = e.to_dev(rand_poly(rng, e.primes, g, e.n, polys=3))
    src = view_at(e, a, 3, len(g), offset, extra)
    want, got = e.torch.empty_like(a), e.torch.empty_like(a)
    e.ntt_(want, a, g)
    e.ntt_(got, src, g)
    assert e.torch.equal(got, want) and e.torch.equal(src, a)
    for cen in (False, True):
        e.intt_(want, got, g, centred=cen)
        dst = view_at(e, e.torch.zeros_like(a), 3, len(g), offset, extra)
        e.intt_(dst, got, g, centred=cen)
        assert e.torch.equal(dst, want)


def test_sides_that_need_a_boundary_are_refused(engine40, pkg):
    """Refused before any launch: the row passes' side off its 16-byte boundary."""
    e = engine40
    g = [0, 20]
    a = e.torch.zeros((2, 2, e.n), dtype=e.torch.int32, device="cuda:0")
    for offset, extra in ((1, 0), (2, 0), (0, 2)):
        off = view_at(e, a, 2, 2, offset, extra)
        with pytest.raises(pkg.CfheError, match="aligned"):
            e.ntt_(off, a, g)
        with pytest.raises(pkg.CfheError, match="aligned"):
            e.intt_(a, off, g)


def test_more_transforms_than_one_launch_covers(engine40):
    """17 polynomials x 40 limbs: 40 transforms past the 640 of one launch pair, out
    of place and in place, against the polynomials on both sides of the seam by
    themselves."""
    e = engine40
    g = e.level_limbs(28)[:40]
    gen = e.torch.Generator(device="cuda:0").manual_seed(17)
    a = e.empty(17, len(g), e.n)
    for i, gi in enumerate(g):
        a[:, i] = e.torch.randint(0, int(e.primes[gi]), (17, e.n), dtype=e.torch.int32, device="cuda:0", generator=gen)
    f, one = e.torch.empty_like(a), e.empty(len(g), e.n)
    e.ntt_(f, a, g)
    for p in (0, 15, 16):
        e.ntt_(one, a[p], g)
        assert e.torch.equal(f[p], one), p
    b = a.clone()
    e.ntt_(b, b, g)
    assert e.torch.equal(b, f)
    back = e.torch.empty_like(a)
    e.intt_(back, f, g, mont_keep=True)
    assert e.torch.equal(back, a)
    e.intt_(b, b, g, mont_keep=True)
    assert e.torch.equal(b, a)
