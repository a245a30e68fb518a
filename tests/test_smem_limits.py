"""A kernel's dynamic shared-memory limit belongs to the device: contexts and host threads share it.  Set to the
size of one launch, it can fall under another context's launch, which is then refused; so it is only ever set to
the device's opt-in maximum or to a constant of the kernel."""
import glob
import os
import re
import threading
import time

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


def test_limits_are_not_one_launch_s():
    sets = []
    for path in sorted(glob.glob(os.path.join(ROOT, "snapi_b200", "csrc", "*.cu*"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"cudaFuncAttributeMaxDynamicSharedMemorySize\s*,\s*([^;]*?)\)\s*[;)!]", src):
            value = re.sub(r"\(int\)|\s", "", m.group(1)).rstrip(")")
            sets.append((os.path.basename(path), value))
            if re.match(r"k[A-Z]\w*$", value):  # the kernel's own constant
                continue
            # a variable that the same file gets from the device, or (raise_smem_limits) is handed that
            assert re.search(r"cudaDeviceGetAttribute\(\s*&%s\s*,\s*cudaDevAttrMaxSharedMemoryPerBlockOptin" % value, src) \
                or re.search(r"raise_smem_limits\(int %s\)" % value, src), sets[-1]
    assert len(sets) >= 5, sets


@pytest.mark.gpu
def test_builds_of_several_threads_are_those_of_one(eos3, config3):
    """One context per host thread, batches whose marches take a different size of shared memory (CTAs of 32
    threads and of 128): every call gives the bits of a single thread's."""
    import snapi_b200 as sb
    from snapi_b200.eos_tables import EosTables
    nodes = config3["nodes"]
    sizes = [500] + [1, 2, 3, 5] * 2  # marches of 500 pixels take four times the shared memory a CTA

    def context():
        ctx = sb.Context.from_fixture(config3, max_batch=512)
        ctx.eos_set(EosTables(eos3))
        return ctx

    def build(ctx, npix):
        rec, _, nt, st = ctx.build_records(nodes[np.arange(npix) % len(nodes)], tangents=False, want_nt=True)
        return rec, nt, st

    ctxs = [context() for _ in sizes]
    want = [build(c, n) for c, n in zip(ctxs, sizes)]
    errors, end = [], time.monotonic() + 8.0

    def run(ctx, npix, ref):
        try:
            while time.monotonic() < end and not errors:
                for a, b in zip(build(ctx, npix), ref):
                    np.testing.assert_array_equal(a, b)
        except Exception as e:  # noqa: BLE001
            errors.append((npix, e))

    threads = [threading.Thread(target=run, args=a) for a in zip(ctxs, sizes, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in ctxs:
        c.close()
    assert not errors, errors
