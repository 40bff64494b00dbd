"""What a server's budget counts of a request's operator set: its smallest budget
that takes the request, found by bisection, covers the FP64 operators and their
fixed-point integers (8 bytes an element each) and does not exceed what a batch
of the same instance holds."""
import pytest

pytestmark = pytest.mark.gpu


def takes(fg, budget, p):
    s = fg.Server(budget)
    try:
        s.submit(p, 1, 5)
        return True
    except fg.FalconError as e:
        assert "budget" in str(e)
        return False


@pytest.mark.parametrize("R,Nm,scheme", [(33, 42, "CNAB2"), (65, 85, "SBDF3"), (49, 30, "ARS443"), (33, 21, "RK2")])
def test_the_smallest_budget(fg, R, Nm, scheme):
    p = fg.make_params(R, Nm, scheme)
    b = fg.Batch([p])
    held = b.device_bytes
    b.close()
    low, high = 1, 4 * held
    assert takes(fg, high, p)
    while high - low > 64:
        mid = (low + high) // 2
        low, high = (low, mid) if takes(fg, mid, p) else (mid, high)
    M = Nm + 1
    per_mode = M * (2 * R + 2) * R if scheme == "RK2" else 4 * M * R * R  # Poisson, or temperature and vorticity solves
    fields = 13 * 16 * R * M                                               # of an instance, at least
    counted = 8 * per_mode * (1 if scheme == "RK2" else 2)
    assert counted + fields <= high <= held + 64, (counted + fields, high, held)
