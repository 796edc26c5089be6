"""Nucleus B has charge amplitudes of its own only where both nuclei's lines
are made at a time. At 1024^2 FP64 a work buffer holds two sheets: with two a
nucleus the lines run side by side, with three they do not, and nothing else
that a context holds differs. The array is 8 MB; the device hands memory out in
pieces of 2 MB, so the two contexts' figures may be off by less than that."""
import pytest
import torch

import ipglasma_b200 as ipg

pytestmark = pytest.mark.gpu


def held(Ny):
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ev = ipg.Event(ipg.Config(size=1024, L=40.0, Ny=Ny, maxtime=0.1, precision=ipg.FP64))
    used = before - torch.cuda.mem_get_info()[0]
    ev.close()
    return used


def test_no_second_amplitude_array_where_the_nuclei_take_turns():
    held(2)
    assert held(2) - held(3) > (8 << 20) - (4 << 20)
