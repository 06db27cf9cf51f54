"""Admission of FP64 requests whose products can go by residues: the residue buffers are
optional, so a budget that holds a request without them accepts it, as many requests run
side by side as without them, and mixed requests are not charged for them. Dry-run slots:
the footprints and admission of a GPU run.

What a request cannot do without is bounded from both sides here: its matrices, Cmm
(nmeas^2), Ctm, and two nmeas x 1,024 panel buffers, plus at most 2 % for geometry."""
import numpy as np
import pytest

import moao_b200 as M
from moao_b200 import params as P
from moao_b200.serve import Server

PROF = (np.array([0.7, 0.3]), np.array([0.0, 8000.0]), np.array([25.0, 25.0]))


@pytest.fixture(scope="module")
def large(tmp_path_factory, built):
    """The files of a 39 m system with 40 subapertures across, and its needed bytes."""
    d = str(tmp_path_factory.mktemp("large"))
    s, a = P.config_scaled(40, 2)
    P.write_system(d, s, a)
    files = d + "/sys-params.txt", d + "/prof-1-atmos-night0.txt"
    t = M.Tomo(*files)
    n, m = t.getNMeas(), t.getNMeasTS()
    return files, 8.0 * (n * n + m * n + 2 * 1024 * n) / 1e9


def server(large, gb, slots=4):
    srv = Server(slots=slots, hbm_budget_gb=gb, dry_run=True)
    return srv, srv.add_system(*large[0])


def test_accepted_without_residues(large):
    need = 1.02 * large[1]
    srv, sid = server(large, need)
    with srv:
        r = srv.wait(srv.submit(sid, *PROF, dry_run_ms=1))
        assert r["status"] == 0 and large[1] < r["footprint_gb"] <= need
        assert srv.stats()["peak_admitted_gb"] <= need


@pytest.mark.parametrize("room", [2.5, 3.2])
def test_as_many_side_by_side(large, room):
    need = 1.02 * large[1]
    srv, sid = server(large, room * need)
    with srv:
        ids = [srv.submit(sid, *PROF, dry_run_ms=80) for _ in range(6)]
        assert all(srv.wait(i)["status"] == 0 for i in ids)
        st = srv.stats()
        assert st["max_in_flight"] == int(room)
        assert st["peak_admitted_gb"] <= st["budget_gb"] + 1e-9


def test_kept_residues_make_room(large):
    """Two requests fit with their residues; what their slots keep of them goes when a
    third slot's request needs the memory."""
    need = 1.02 * large[1]
    srv, sid = server(large, 3.1 * need, slots=3)
    with srv:
        assert srv.wait(srv.submit(sid, *PROF, dry_run_ms=1))["status"] == 0
        ids = [srv.submit(sid, *PROF, dry_run_ms=80) for _ in range(3)]
        assert all(srv.wait(i)["status"] == 0 for i in ids)
        st = srv.stats()
        assert st["max_in_flight"] == 3
        assert st["peak_admitted_gb"] <= st["budget_gb"] + 1e-9


def test_admitted_with_residues_where_there_is_room(large):
    srv, sid = server(large, 1000.0, slots=1)
    with srv:
        r = srv.wait(srv.submit(sid, *PROF, dry_run_ms=1))
        assert srv.stats()["peak_admitted_gb"] > 1.1 * r["footprint_gb"]
        # a mixed request on the same slot keeps them, one after it is FP64 again
        for prec in ("mixed", "fp64"):
            assert srv.wait(srv.submit(sid, *PROF, prec=prec, dry_run_ms=1))["status"] == 0
