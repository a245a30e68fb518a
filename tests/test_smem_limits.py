"""A kernel's dynamic shared-memory limit belongs to the device: contexts and host threads share it.  Set to the
size of one launch, it can fall under another context's launch, which is then refused; so it is only ever set to
the device's opt-in maximum or to a constant of the kernel."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_a_coarser_width_in_another_context_leaves_this_one_s_launch(config3):
    """Broadening on a fine grid (150 KB of shared memory a CTA) before and after another context broadens on a
    coarse one."""
    import snapi_b200 as sb
    lam = np.asarray(config3["lambda_air"])
    span = lam[-1] - lam[0]
    a, b = sb.Context.from_fixture(config3, max_batch=8), sb.Context.from_fixture(config3, max_batch=8)
    spectra = config3["stokes"][:4]
    want = a.broaden(spectra, 2.0 * span / 4550)  # 4591 points of half a width over the span and 10 widths a side
    b.broaden(spectra, span / 20)
    np.testing.assert_array_equal(a.broaden(spectra, 2.0 * span / 4550), want)
    a.close()
    b.close()
