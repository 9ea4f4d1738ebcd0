"""Contexts in different host threads: a call of one thread does not depend on
what another thread's context calls at the same time (a context itself belongs
to one thread at a time).  Fields of different sizes share kernels, so a kernel
attribute set for one field's size must hold for every other."""

import threading

import numpy as np
import pytest

import gks_ic

pytestmark = pytest.mark.gpu


def together(calls, rounds):
    """Each call repeated in a thread of its own, until one fails or the last has done its rounds."""
    stop, errors = threading.Event(), []

    def work(call, n):
        try:
            done = 0
            while not stop.is_set() and (n is None or done < n):
                call()
                done += 1
        except Exception as e:  # noqa: BLE001 - reported by the test
            errors.append(e)
        finally:
            if n is not None or errors:
                stop.set()

    threads = [threading.Thread(target=work, args=(c, n)) for c, n in zip(calls, [None] * (len(calls) - 1) + [rounds])]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def field(gks, nc, particles=0):
    case = gks_ic.make_dhit(nc, k0=min(4.0, nc / 4), Mt=0.4, seed=nc)
    s = gks.Solver(gks.phys_from_case(case))
    s.upload(gks_ic.to_conservative_padded(case))
    if particles:
        s.particles_locate(*(np.random.default_rng(nc).random((3, particles)) * (2 * np.pi)))
    return s


@pytest.mark.parametrize("what", ["particles", "stats"])
def test_two_sizes_in_two_threads(gks, what):
    """A small field and one whose lines need far more shared memory, the larger
    one's results the same as alone."""
    sizes = (8, 160) if what == "particles" else (8, 200)
    small, large = (field(gks, nc, 100 if what == "particles" else 0) for nc in sizes)
    with small, large:
        def call(s):
            if what == "particles":
                s.particles_props()
                return s.particles_get()
            return s.stats_array()

        alone = call(large)
        got = []
        errors = together([lambda: call(small), lambda: got.append(call(large))], 400)
        assert not errors, errors[0]
        assert all(np.array_equal(g, alone) for g in got)
