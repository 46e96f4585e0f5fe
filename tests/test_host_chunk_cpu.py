"""CPU test of the host-buffer products' default chunk: its device workspace (three
slots of a, b and c, and the chunk's spectra) follows 80 MiB of spectra per chunk,
not the device product's larger waves."""
import pytest


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n_power", [14, 15, 16, 17, 18, 20])
def test_default_chunk_workspace_is_bounded(gf, n_power, bits):
    # spectra of a chunk: 2 N/2 complex = 2 reals per coefficient; a slot: 3 reals
    spectra = 80 << 20
    slots = 3 * 3 * spectra // 2
    need = gf.lib().gpufft_negacyclic_mul_host_workspace_bytes(n_power, 1 << 20, 0, bits)
    assert 0 < need <= spectra + slots + 9 * 256  # every buffer of a slot is rounded up to 256 bytes
