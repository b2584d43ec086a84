"""An iteration's last kernel writes its record to the integrator's pinned memory, which
the allocator of pinned memory knows nothing of: no call may end, by an exception either,
with such a kernel in flight, or the memory could be another tensor's by then."""
import pytest
import torch

import vegas_gb300 as vg
from vegas_gb300.ravg import RAvg

pytestmark = pytest.mark.gpu


class Stop(BaseException):
    """As KeyboardInterrupt: not caught by handlers of Exception."""


@pytest.mark.parametrize('name', ['converged', 'add'])
def test_exceptions_leave_no_iteration_in_flight(name, monkeypatch):
    f = vg.Gaussian(a=100.0, c=0.5, dim=4)
    I = vg.Integrator(4 * [[0, 1]], neval=30000000, seed=1)
    I(f, nitn=1)
    torch.cuda.synchronize()

    def stop(self, *args, **kargs):
        raise Stop

    monkeypatch.setattr(RAvg, name, stop)
    with pytest.raises(Stop):
        I(f, nitn=5, rtol=1e-9)
    idle = torch.cuda.current_stream().query()
    torch.cuda.synchronize()
    assert idle
    monkeypatch.undo()
    assert abs(I(f, nitn=2, rtol=0).mean - 1.0) < 0.01
