"""GPU parity of the RK3 stage against the oracle, through the C ABI.

FP64 tolerance: after one stage the GPU and the oracle agree to 1e-11 of the
field scale; after a few steps to 1e-9 (the two evaluate the same
expressions in a different order: fused spectral derivatives and a
level-parallel z-sweep instead of 1D transforms and ring buffers).  The
mixed form is held to an FP32 envelope of the FP64 oracle.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def relerr(a, b, scale=None):
    s = np.abs(b).max() if scale is None else scale
    return np.abs(a - b).max() / max(s, 1e-300)


def make_pair(product, nx, ny, nz, precision=8, seed=7, amp=0.3, dt=2e-3, **kw):
    cfg_o = O.make_config(nx, ny, nz, dt=dt, **kw)
    o = O.Oracle(cfg_o)
    o.make_ic(seed=seed, amp=amp)
    f = o.get_fields()
    cfg_g = product.channel_config(nx, ny, nz, dt=dt, precision=precision,
                                   imodel=kw.get("imodel", 3), isurface=kw.get("isurface", 6),
                                   tke_production=kw.get("tke_production", 0))
    cfg_g.z0 = cfg_o.z0
    g = product.LesGpu(cfg_g)
    g.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
    return o, g, f


def compare(o, g, tol_f, tol_t, label=""):
    fo, to_ = o.get_fields(), o.get_tendencies()
    fg, tg = g.download(), g.download_tendencies()
    vscale = np.abs(fo["u"]).max()
    errs = {}
    for k in "uvw":
        errs[k] = relerr(fg[k], fo[k], vscale)
    errs["e"] = relerr(fg["e"], fo["e"])
    rscale = max(np.abs(to_["ru"]).max(), np.abs(to_["rv"]).max(), np.abs(to_["rw"]).max())
    for k in ("ru", "rv", "rw"):
        errs[k] = relerr(tg[k], to_[k], rscale)
    errs["re"] = relerr(tg["re"], to_["re"])
    errs["p"] = relerr(fg["p"], fo["p"])
    bad = {k: v for k, v in errs.items() if v > (tol_f if k in "uvwe" else tol_t)}
    assert not bad, (label, errs)
    return errs


@pytest.mark.parametrize("case", [
    dict(nx=16, ny=16, nz=8, imodel=3, isurface=6, tke_production=0),
    dict(nx=16, ny=16, nz=8, imodel=4, isurface=1, tke_production=1),
    dict(nx=32, ny=16, nz=12, imodel=3, isurface=1, tke_production=1),
    dict(nx=16, ny=32, nz=6, imodel=3, isurface=6, tke_production=1),
    # the other wall models (lowerbc.f90:126-161, upperbc.f90:124-158)
    dict(nx=16, ny=16, nz=8, imodel=3, isurface=2, tke_production=0),
    dict(nx=32, ny=16, nz=8, imodel=3, isurface=3, tke_production=0),
    dict(nx=16, ny=16, nz=8, imodel=3, isurface=4, tke_production=1),
    dict(nx=16, ny=32, nz=8, imodel=4, isurface=5, tke_production=0),
], ids=lambda c: "{nx}x{ny}x{nz}-m{imodel}-s{isurface}-p{tke_production}".format(**c))
def test_one_stage_then_two_steps_fp64(gpu_lib, product, case):
    kw = dict(case)
    nx, ny, nz = kw.pop("nx"), kw.pop("ny"), kw.pop("nz")
    o, g, _ = make_pair(product, nx, ny, nz, **kw)
    o.stage(0, 1, 1)
    g.stage(0, True, 1)
    compare(o, g, 1e-11, 1e-9, "stage1")
    for s in (2, 3):
        o.stage(0, 1, s)
        g.stage(0, True, s)
    compare(o, g, 1e-11, 1e-9, "step1")
    for it in (1,):
        for s in (1, 2, 3):
            o.stage(it, 1, s)
            g.stage(it, True, s)
    compare(o, g, 1e-10, 1e-8, "step2")
    g.sync()


def test_split_entry_points_match_fused_stage(gpu_lib, product):
    o, g, f = make_pair(product, 32, 32, 16)
    cfg = g.cfg
    g2 = product.LesGpu(cfg)
    g2.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
    for it in range(2):
        for s in (1, 2, 3):
            g.stage(it, True, s)
            g2.stage_split(it, True, s)
    a, b = g.download(), g2.download()
    for k in "uvwep":
        assert relerr(b[k], a[k]) < 1e-12, k
    ta, tb = g.download_tendencies(), g2.download_tendencies()
    for k in ta:
        # re is a small residual of nearly cancelling TKE budget terms
        assert relerr(tb[k], ta[k]) < (1e-9 if k == "re" else 1e-11), k


def test_graph_step_matches_stages(gpu_lib, product):
    o, g, f = make_pair(product, 32, 32, 16)
    g2 = product.LesGpu(g.cfg)
    g2.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
    for it in range(3):
        for s in (1, 2, 3):
            g.stage(it, False, s)
        g2.step(it=it + 1, mnout=False)
    g2.sync()
    a, b = g.download(), g2.download()
    for k in "uvwep":
        assert np.array_equal(a[k], b[k]), k  # same kernels, deterministic reductions
    assert g2.kernel_launches() > 0


@pytest.mark.parametrize("imodel,tke", [(3, 0), (3, 1)])
def test_initial_field_and_statistics_are_reproducible(gpu_lib, product, imodel, tke):
    """make_ic's plane means and compmn's divz / SGS-mean rows are per-block
    partial sums reduced in a fixed order: two handles stepping the same
    field agree bit for bit (fused row kernel and, with TKE production, the
    unfused k_flux path)."""
    out = []
    for _ in range(2):
        cfg = product.channel_config(32, 32, 16, dt=2e-3, re_tau=180.0, imodel=imodel, tke_production=tke)
        g = product.LesGpu(cfg)
        g.make_ic(seed=5, amp=0.2, re_tau=180.0)
        for it in range(3):
            g.step(it=it, mnout=True)
        g.sync()
        out.append((g.download(), g.stats()))
        g.close()
    (fa, (ma, sa)), (fb, (mb, sb)) = out
    for k in "uvwep":
        assert np.array_equal(fa[k], fb[k]), k
    assert np.array_equal(ma, mb) and np.array_equal(sa, sb)
    assert np.abs(ma[13:19]).max() > 0 and ma[2].max() > 0


def test_profile_stage_names_every_kernel(gpu_lib, product):
    """The per-kernel trace of one stage resolves every launch (internal
    linkage kernels such as k_wall_final included) to its les:: kernel name."""
    o, g, f = make_pair(product, 32, 32, 16)
    prof = g.profile_stage(2)
    names = [n for n, _ in prof]
    assert len(names) > 5
    assert all(n.startswith("k_") for n in names), names
    assert "k_wall_final" in names and any(n.startswith("k_row_fused") for n in names), names
    assert all(t >= 0 for _, t in prof)


def test_c1_ten_steps_fp64(gpu_lib, product):
    """Config 1 (64^3, Re_tau 180, Deardorff, isurface 6): 10 RK3 steps."""
    cfg_o = O.make_config(64, 64, 64, dt=1e-3, re_tau=180.0)
    o = O.Oracle(cfg_o)
    o.make_ic(seed=12345, amp=0.1)
    dt = o.cfl_dt(0.5)
    o.set_dt(dt)
    f = o.get_fields()
    cfg_g = product.channel_config(64, 64, 64, dt=dt, re_tau=180.0)
    g = product.LesGpu(cfg_g)
    g.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
    o.step(0, 10, 5)
    for it in range(10):
        g.step(it=it, mnout=(it % 5 == 0), dt=dt)
    g.sync()
    errs = compare(o, g, 1e-10, 1e-8, "C1 10 steps")
    o.compmn()  # the reference computes the moments only at mnout steps
    mo, so = o.stats()
    mg, sg = g.stats()
    for r in (0, 1, 3, 4, 6, 7, 8, 9, 10, 11, 17, 18):
        assert relerr(mg[r], mo[r], max(np.abs(mo[r]).max(), 1e-12)) < 1e-8, r
    assert np.abs(mg[5]).max() < 1e-15 and np.abs(mo[5]).max() < 1e-15  # wxym: zero to round-off
    np.testing.assert_allclose(sg[:4], so[:4], rtol=1e-9, atol=1e-15)


@pytest.mark.parametrize("n", [192, 256, 384, 512])
def test_fused_row_plans_at_production_widths(gpu_lib, product, n):
    """The fused row kernel's three-pass Stockham plans of the production
    grids (padded rows 288, 384, 576 and 768) against the oracle, one stage
    in each precision (nz = 4 keeps the oracle to seconds); the stage tests
    above cover the two-pass plans of the small grids."""
    o, g, _ = make_pair(product, n, n, 4, amp=0.3)
    o.stage(0, 1, 1)
    g.stage(0, True, 1)
    compare(o, g, 1e-11, 1e-9, "fp64 %d" % n)
    o, g, _ = make_pair(product, n, n, 4, precision=4, amp=0.3)
    o.stage(0, 1, 1)
    g.stage(0, True, 1)
    fo, fg = o.get_fields(), g.download()
    vscale = np.abs(fo["u"]).max()
    for k in "uvw":
        assert relerr(fg[k], fo[k], vscale) < 2e-5, (n, k)
    assert relerr(fg["e"], fo["e"]) < 2e-5, n


@pytest.mark.parametrize("nx,ny,nz", [(16, 32, 4), (32, 16, 9), (64, 16, 5), (96, 32, 7), (128, 16, 5), (192, 16, 5),
                                      (256, 16, 4), (384, 16, 4), (512, 16, 5)])
def test_fused_row_plans_with_clipped_tke(gpu_lib, product, nx, ny, nz):
    """Every row plan of the fused kernel (padded rows 24 to 768, odd level
    counts) with a TKE whose expansion the floor clips: the correction terms
    are read at the permuted position of each point.  Tolerances of the
    unclipped stage tests."""
    rng = np.random.default_rng(nx + nz)
    e = 1e-3 * rng.random((nz, ny, nx)) ** 4
    for precision, tol in ((8, 1e-11), (4, 2e-5)):
        o, g, f = make_pair(product, nx, ny, nz, precision=precision, amp=0.3)
        o.set_fields(e=e)
        o.deal_fields()
        f = o.get_fields()
        g.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
        for s in (1, 2):
            o.stage(0, 1, s)
            g.stage(0, True, s)
        fo, fg = o.get_fields(), g.download()
        vscale = np.abs(fo["u"]).max()
        for k in "uvw":
            assert relerr(fg[k], fo[k], vscale) < tol, (precision, k)
        assert relerr(fg["e"], fo["e"]) < tol, precision


def test_mixed_precision_envelope(gpu_lib, product):
    o, g, f = make_pair(product, 64, 64, 32, precision=4, amp=0.1)
    for it in range(3):
        for s in (1, 2, 3):
            o.stage(it, 1, s)
            g.stage(it, True, s)
    fo, fg = o.get_fields(), g.download()
    vscale = np.abs(fo["u"]).max()
    for k in "uvw":
        assert relerr(fg[k], fo[k], vscale) < 2e-5, k
    # the mean profile comes from the FP64 shadow of the kx=ky=0 mode
    o.compmn()
    mo, _ = o.stats()
    mg, _ = g.stats()
    assert relerr(mg[3], mo[3]) < 1e-6


def test_gpu_ic_is_divergence_free_and_matches_oracle(gpu_lib, product):
    nx, ny, nz = 64, 64, 32
    cfg_o = O.make_config(nx, ny, nz, dt=1e-3, re_tau=395.0)
    o = O.Oracle(cfg_o)
    o.make_ic(seed=12345, amp=0.1, re_tau=395.0)
    g = product.LesGpu(product.channel_config(nx, ny, nz, dt=1e-3, re_tau=395.0))
    g.make_ic(seed=12345, amp=0.1, re_tau=395.0)
    fo, fg = o.get_fields(), g.download()
    for k in "uvwe":
        assert relerr(fg[k], fo[k], np.abs(fo["u"]).max()) < 1e-12, k
    assert abs(g.cfl_dt(0.5) - o.cfl_dt(0.5)) < 1e-12 * o.cfl_dt(0.5)


def test_spectra_match_oracle(gpu_lib, product):
    o, g, f = make_pair(product, 32, 32, 8)
    for field in range(4):
        zo, z2o = o.spectra(field, 3)
        zg, z2g = g.spectra(field, 3)
        assert relerr(zg, zo) < 1e-11, field
        assert relerr(z2g, z2o) < 1e-11, field


def test_nan_in_state_is_reported(gpu_lib, product):
    """Fault injection on the host: a NaN planted in an uploaded field makes
    the next step report LES_ENAN instead of continuing silently."""
    o, g, f = make_pair(product, 16, 16, 8)
    u = f["u"].copy()
    u[3, 5, 7] = np.nan
    g.upload(u, f["v"], f["w"], f["e"], f["p"])
    g.step(it=1)
    with pytest.raises(product.LesError) as ei:
        g.sync()
    assert ei.value.code == product.LES_ENAN


def test_out_of_order_split_calls_are_rejected(gpu_lib, product):
    o, g, f = make_pair(product, 16, 16, 8)
    with pytest.raises(product.LesError) as ei:
        g.press()
    assert ei.value.code == product.LES_ESTATE


@pytest.mark.parametrize("nz", [4, 5, 9, 63, 64, 65, 127, 128, 129, 255, 256, 257, 512, 513])
def test_pressure_columns_of_every_chunk_length(gpu_lib, product, nz):
    """The chunked pressure solve and update at the edges of its chunk lengths
    (2, 4, 8 levels), of its last chunk, and of the one-thread sweep beyond
    512 levels; fields, tendencies and p against the oracle, and divergence at
    round-off (the tolerances of the stage tests)."""
    o, g, _ = make_pair(product, 16, 16, nz, dt=2e-4)
    for s in (1, 2):
        o.stage(0, 1, s)
        g.stage(0, True, s)
    compare(o, g, 1e-11, 1e-9, "nz %d" % nz)
    g2 = product.LesGpu(g.cfg)
    f = g.download()
    g2.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
    g.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
    g.stage(0, True, 1)
    g2.stage_split(0, True, 1)
    a, b = g.download(), g2.download()
    for k in "uvwep":
        assert relerr(b[k], a[k]) < 1e-12, k


@pytest.mark.parametrize("nx,ny,nz,imodel", [(96, 128, 45, 4), (128, 128, 20, 3), (128, 96, 33, 3)])
def test_pressure_columns_in_wide_blocks(gpu_lib, product, nx, ny, nz, imodel):
    """Grids with enough columns for the pressure solve's wide blocks, through
    the whole stage and the six entry points: what the solve and its update
    write (u, v, w, p and their tendencies), to the tolerances of the stage
    tests."""
    o, g, f = make_pair(product, nx, ny, nz, imodel=imodel)
    g2 = product.LesGpu(g.cfg)
    g2.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
    o.stage(0, 1, 1)
    g.stage(0, True, 1)
    g2.stage_split(0, True, 1)
    fo, to_ = o.get_fields(), o.get_tendencies()
    vscale = np.abs(fo["u"]).max()
    rscale = max(np.abs(to_[k]).max() for k in ("ru", "rv", "rw"))
    for h in (g, g2):
        fg, tg = h.download(), h.download_tendencies()
        for k in "uvw":
            assert relerr(fg[k], fo[k], vscale) < 1e-11, k
        for k in ("ru", "rv", "rw"):
            assert relerr(tg[k], to_[k], rscale) < 1e-9, k
        assert relerr(fg["p"], fo["p"]) < 1e-9


@pytest.mark.parametrize("clipped", [False, True])
@pytest.mark.parametrize("nx,ny,nz,imodel,tke", [(16, 32, 4, 4, 0), (96, 128, 5, 4, 1), (96, 128, 8, 3, 1), (128, 96, 13, 4, 0)])
def test_flux_columns_of_the_unfused_stage(gpu_lib, product, nx, ny, nz, imodel, tke, clipped):
    """k_flux with one level, several levels and a short last chunk per thread
    (padded planes of 216 point blocks), and the clip kernels with a TKE that
    they leave alone and one that they raise.  Tolerances of the unclipped stage
    tests; e in FP64 only (white noise in e rounds to 2e-5 of it in FP32, by the
    advective term, whichever way the fluxes are computed)."""
    rng = np.random.default_rng(nx + nz)
    e = 1e-3 * rng.random((nz, ny, nx)) ** 4 if clipped else 1e-3 * (1.0 + 0.1 * rng.random((nz, ny, nx)))
    for precision, tol in ((8, 1e-11), (4, 2e-5)):
        o, g, f = make_pair(product, nx, ny, nz, precision=precision, amp=0.3, imodel=imodel, tke_production=tke)
        o.set_fields(e=e)
        o.deal_fields()
        f = o.get_fields()
        g.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
        for s in (1, 2):
            o.stage(0, 1, s)
            g.stage(0, True, s)
        fo, fg = o.get_fields(), g.download()
        vscale = np.abs(fo["u"]).max()
        for k in "uvw":
            assert relerr(fg[k], fo[k], vscale) < tol, (precision, k)
        if precision == 8:
            assert relerr(fg["e"], fo["e"]) < tol


@pytest.mark.parametrize("nx,ny,imodel", [(16, 16, 3), (512, 16, 3), (512, 128, 3), (128, 64, 4)])
def test_statistics_from_few_and_many_partial_sums(gpu_lib, product, nx, ny, imodel):
    """divz and the SGS means from 9, 288, 2304 (one partial sum per warp of
    k_row_fused) and 576 (k_flux) partials a level: less than one round of
    k_sum_parts' threads, a remainder and several unrolled rounds.  A field
    with a divergence, so that divz is no round-off; one stage from the same
    field, tolerance that of one stage's tendencies (1e-9 of the scale)."""
    o, g, f = make_pair(product, nx, ny, 4, imodel=imodel)
    o.set_fields(u=f["u"] + 0.5 * np.sin(2 * np.pi * np.arange(nx) / nx)[None, None, :])
    o.deal_fields()
    f = o.get_fields()
    g.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
    o.stage(0, 1, 1)
    g.stage(0, True, 1)
    o.compmn()
    mo, _ = o.stats()
    mg, _ = g.stats()
    assert mo[2].min() > 1e-3
    assert relerr(mg[2], mo[2]) < 1e-9
    scale = np.abs(mo[13:19]).max()
    for r in range(13, 19):
        assert relerr(mg[r], mo[r], scale) < 1e-9, r


@pytest.mark.parametrize("nz", [4, 8, 9, 33, 70, 99])
def test_pressure_columns_on_large_planes(gpu_lib, product, nz):
    """The pressure solve where a plane's columns fill the device: chunks of 4
    and 8 levels, one chunk, a short last one, the columns split for two blocks
    per SM (70 and 99 levels), blocks of 16 and 32 modes, the whole
    stage and the six entry points.  Tolerances of the stage tests."""
    for precision, tol in ((8, 1e-11), (4, 2e-5)):
        o, g, f = make_pair(product, 192, 128, nz, precision=precision)
        g2 = product.LesGpu(g.cfg)
        g2.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
        for s in (1, 2):
            o.stage(0, 1, s)
            g.stage(0, True, s)
            g2.stage_split(0, True, s)
        fo = o.get_fields()
        vscale = np.abs(fo["u"]).max()
        for h in (g, g2):
            fg = h.download()
            for k in "uvw":
                assert relerr(fg[k], fo[k], vscale) < tol, (precision, k)
            if precision == 8:
                assert relerr(fg["p"], fo["p"]) < 1e-9
            h.close()


@pytest.mark.parametrize("clipped", [False, True])
@pytest.mark.parametrize("nx,ny,nz,imodel,tke", [(16, 32, 4, 4, 0), (96, 128, 5, 4, 1), (96, 128, 8, 3, 1), (128, 96, 13, 4, 0)])
def test_tke_fluxes_of_the_unfused_stage_in_fp32(gpu_lib, product, nx, ny, nz, imodel, tke, clipped):
    """e after two stages of the unfused middle in FP32: its fluxes, the shear
    production and the clip corrections.  A smooth e, which rounding leaves
    alone: 4 units in the last place on u, v, w and e move the oracle's e by
    2.4e-7 to 2.9e-7 of its maximum on these inputs, the stages by 0.6 to 44 per
    cent.  The bound is 16 times the former."""
    o, g, _ = make_pair(product, nx, ny, nz, precision=4, amp=0.3, imodel=imodel, tke_production=tke)
    x, y, z = 2 * np.pi * np.arange(nx) / nx, 2 * np.pi * np.arange(ny) / ny, (np.arange(nz) + 0.5) / nz
    wave = (np.cos(x)[None, None, :] * np.cos(2 * y)[None, :, None]) * (1 + 0.3 * np.cos(np.pi * z))[:, None, None]
    o.set_fields(e=1e-3 * ((0.5 if clipped else 1.5) + wave))
    o.deal_fields()
    f = o.get_fields()
    g.upload(f["u"], f["v"], f["w"], f["e"], f["p"])
    for s in (1, 2):
        o.stage(0, 1, s)
        g.stage(0, True, s)
    fo, fg = o.get_fields(), g.download()
    assert (np.abs(fo["e"] - 1e-6).min() < 1e-9) == clipped
    assert relerr(fg["e"], fo["e"]) < 16 * 2.9e-7
