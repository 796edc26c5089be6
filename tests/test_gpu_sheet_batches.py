"""Sheet batches of the Wilson-line stage and of its adjoint, around the sizes
where a nucleus's sheets stop being one batch (256^2: 32 sheets a work buffer
in FP64; the two nuclei then no longer run side by side), and the spectrum's
fold over few blocks.

Bounds: V is a product of Ny unitary matrices, each within 1e-14 of the same
exponential, so 1e-12 between two evaluations of one product; g2mu_bar and its
restatement sum the same 8 Ny products in different order, 1e-12 of the sum of
their magnitudes; counts are exact."""
import numpy as np
import pytest

import ipglasma_b200 as ipg
from ipglasma_b200.synthetic import gaussian_blobs

pytestmark = pytest.mark.gpu


def event(N, Ny, seed=5, **more):
    L = N * 0.078125
    ev = ipg.Event(ipg.Config(size=N, L=L, Ny=Ny, maxtime=0.05, seed=seed, **more))
    A, B = gaussian_blobs(N, L)
    ev.set_g2mu(A, B)
    ev.use_device_noise()
    return ev, np.stack([A, B])


@pytest.mark.parametrize("N,Ny,prec", [(8, 1, 0), (64, 3, 1), (256, 31, 0), (256, 32, 0),
                                       (256, 33, 0), (256, 65, 1)])
def test_nuclei_give_the_same_lines_in_either_order(N, Ny, prec):
    """Exchanging the nuclei (maps and noise) exchanges V_A and V_B to the bit,
    whichever stream and buffer each was made on."""
    ev, g = event(N, Ny, precision=prec)
    xi = [ev.draw_device_noise(k) for k in range(2)]
    ev.init_fields(allow_nonconverged=True)
    drawn = [ev.get_field(f) for f in (ipg.VA, ipg.VB)]
    lines = []
    for order in ((0, 1), (1, 0)):
        ev.set_g2mu(g[order[0]], g[order[1]])
        ev.set_noise(xi[order[0]].ravel(), xi[order[1]].ravel())
        ev.init_fields(allow_nonconverged=True)
        lines.append([ev.get_field(f) for f in (ipg.VA, ipg.VB)])
    ev.close()
    for k in range(2):
        assert np.array_equal(lines[0][k], lines[1][1 - k])
        assert np.array_equal(lines[0][k], drawn[k])
        V = lines[0][k]
        assert np.abs(V @ V.conj().transpose(0, 2, 1) - np.eye(3)).max() < 1e-12


@pytest.mark.parametrize("N,Ny", [(32, 1), (64, 5), (256, 32), (256, 35)])
def test_map_gradient_is_the_sum_over_the_charges(N, Ny):
    """rho = g sqrt(g2mu / Ny) xi, so g2mu_bar = sum_k,a rho_bar xi g / (2 sqrt(g2mu Ny))."""
    ev, g = event(N, Ny, newton_tolerance=1e-12)
    xi = np.stack([ev.draw_device_noise(k) for k in range(2)])
    ev.init_fields(allow_nonconverged=True)
    ev.forward(1)
    grad = ev.backward(1.0, 0.0, inputs=True, rho=True)
    ev.close()
    w = 2.0 / (2 * np.sqrt(g * Ny))
    want = (grad["rho"] * xi).sum(axis=(1, 3)) * w
    size = np.abs(grad["rho"] * xi).sum(axis=(1, 3)) * w
    assert np.abs(grad["g2mu"]).max() > 0
    assert np.all(np.abs(grad["g2mu"] - want) <= 1e-12 * size)


@pytest.mark.parametrize("N", [8, 16, 32, 64])
def test_spectrum_counts_every_momentum_once(N):
    ev, _ = event(N, 2)
    ev.init_fields(allow_nonconverged=True)
    ev.evolve(1)
    m = ev.multiplicity(max_gauge_iterations=20)
    ev.close()
    s = np.sin(np.pi * (-0.5 + np.arange(N) / N))[1:]
    kt = np.sqrt(4 * (s[:, None] ** 2 + s[None] ** 2)).ravel()
    edges = np.arange(ipg.KT_BINS + 1) * (2.83 / ipg.KT_BINS)
    clear = np.abs(kt[:, None] - edges).min(axis=1) > 1e-12  # not on a bin's edge
    low = np.histogram(kt[clear], edges)[0]
    assert m["count_kt"].sum() <= kt.size
    assert np.all(m["count_kt"] >= low)
    assert (m["count_kt"] - low).sum() <= (~clear).sum()
    assert np.isfinite(m["n_kt"]).all() and m["dNdy"] > 0
