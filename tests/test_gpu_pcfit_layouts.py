"""The pattern-centre correlation from planes and from quads, for detectors of
the tensor-memory kernel and of the one for large detectors: the same spectra,
the maxima of the float64 FFT formulation from both, two launches into one
batch included; and a fit on a large enlarged detector through the kernels
and through cuFFT."""

import pytest
import torch

from ebsdtorch_b200._capi import call, load, ptr

pytestmark = pytest.mark.gpu
DEV = "cuda"
SIZES = [(2, 2), (14, 13), (16, 16), (23, 22), (78, 78), (96, 96), (97, 97), (104, 100), (120, 120), (127, 64),
         (64, 127), (127, 127)]


def _stages(sims, pats, hp, wp, suffix):
    n, B = sims.shape[0], pats.shape[0]
    size = int(load().ebsd_pcfit_xcorr_table_bytes(hp, wp))
    tables = torch.empty((size,), dtype=torch.uint8, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    call("ebsd_pcfit_xcorr_tables", hp, wp, ptr(tables), size, None)
    spec_len = 4 * (hp // 2 + 1) * (wp // 2 + 1)
    spec, pspec = torch.empty((n, spec_len), device=DEV), torch.empty((B, spec_len), device=DEV)
    terms = torch.empty_like(pspec)
    for img, out in ((sims, spec), (pats, pspec)):
        call("ebsd_pcfit_spectra" + suffix, ptr(img), hp * wp, img.shape[0], hp, wp, ptr(tables), ptr(out),
             ptr(status), None)
    call("ebsd_pcfit_pattern_terms" + suffix, ptr(pspec), B, hp, wp, ptr(terms), None)
    keys = torch.zeros((B * hp * wp,), dtype=torch.int64, device=DEV)
    for a, b in ((0, 20), (20, n)):
        part = spec[a:b].contiguous()
        call("ebsd_pcfit_xcorr_max" + suffix, ptr(part), b - a, ptr(terms), B, hp, wp, ptr(tables), ptr(keys), a,
             ptr(status), None)
    best = torch.full((B, hp, wp), -1e30, device=DEV)
    index = torch.full((B, hp, wp), -1, dtype=torch.int64, device=DEV)
    call("ebsd_pcfit_fold", ptr(keys), keys.numel(), ptr(best), ptr(index), None)
    assert int(status.item()) == 0
    return spec, terms, best, index


@pytest.mark.parametrize("hp,wp", SIZES)
def test_both_layouts_match_the_fft(hp, wp):
    n, B = 37, 3
    g = torch.Generator().manual_seed(hp * 131 + wp)
    sims = torch.rand((n, hp, wp), generator=g).to(DEV)
    pats = torch.randn((B, hp, wp), generator=g).to(DEV)
    spec, terms, best, index = _stages(sims, pats, hp, wp, "")
    spec_q, terms_q, best_q, index_q = _stages(sims, pats, hp, wp, "_quads")
    h2, wf = hp // 2 + 1, wp // 2 + 1
    for planes, quads in ((spec, spec_q), (terms, terms_q)):
        assert torch.equal(planes.view(-1, 4, h2, wf).permute(0, 2, 3, 1), quads.view(-1, h2, wf, 4))
    sf, pf = torch.fft.rfft2(sims.double()), torch.fft.rfft2(pats.double()).conj()
    maps = torch.fft.fftshift(torch.fft.irfft2(sf[:, None] * pf[None], s=(hp, wp)), dim=(-2, -1))
    v, i = maps.max(dim=0)
    top2, rms = maps.topk(2, dim=0).values, maps.pow(2).mean().sqrt()
    # a 3-term bf16 split is off by about 3e-5 of the maps' RMS (standard deviation)
    clear = top2[0] - top2[1] > 2e-3 * rms
    for b, ix in ((best, index), (best_q, index_q)):
        assert float((b.double() - v).abs().max() / rms) < 2e-4
        assert bool((ix == i)[clear].all())
    if not load().ebsd_pcfit_xcorr_takes_quads(hp, wp):
        assert torch.equal(best, best_q) and torch.equal(index, index_q)  # one kernel, the same arithmetic


def test_fit_on_a_large_detector(monkeypatch):
    from ebsdtorch_b200 import synthetic
    from ebsdtorch_b200.ebsd import EBSDGeometry, MasterPattern, spatial_fft_pc_fitter
    from ebsdtorch_b200.ebsd import fitting as F

    mp_t = synthetic.synthetic_master_pattern(257, seed=5, device=DEV)
    geom = EBSDGeometry((90, 90), tilts_degrees=(0.0, 70.0, 0.0), proj_center=(0.48, 0.52, 0.55))
    q = synthetic.random_quaternions(4, 11).to(DEV)
    pats = synthetic.synthetic_patterns(mp_t, geom, q, mean_counts=300.0, seed=12).view(4, 1, 90, 90)
    mp = MasterPattern(mp_t, laue_group=11)
    kw = dict(pc_x_min=0.4, pc_x_max=0.6, pc_y_min=0.4, pc_y_max=0.6, pc_z_min=0.5, pc_z_max=0.6, pc_z_steps=2,
              dictionary_resolution_deg=6.0, dictionary_indexing_batch_size=256)
    sizes, out, layout = [], {}, F.spectra_layout
    monkeypatch.setattr(F, "spectra_layout", lambda h, w: sizes.append((h, w)) or layout(h, w))
    for path in ("dft", "fft"):
        if path == "fft":
            monkeypatch.setattr(F, "xcorr_supported", lambda hp, wp: False)
        torch.manual_seed(1)
        out[path] = spatial_fft_pc_fitter(mp, pats.clone(), **kw)
    (size,) = sizes
    assert 97 <= min(size) and max(size) <= 127 and layout(*size) == ""
    assert all(torch.equal(a, b) for a, b in zip(out["dft"], out["fft"]))
