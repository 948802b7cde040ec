"""Device memory of the canonical int32 plans' tables."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from test_parity_gpu import gb, root_for  # noqa: E402,F401

Q32 = 998244353
TABLE_BYTES = 5     # GBNTT_Q_TABLE_BYTES


def table_bytes(gb, kind, L, flags=1):  # noqa: F811
    return gb.Plan(kind, 1 << L, Q32, root_for(Q32, 1 << L), 0, flags).query(TABLE_BYTES)


def test_no_one_cta_table_where_every_call_takes_two_passes(gb):  # noqa: F811
    """2^15 and the inverse of 2^14 hold the tables of the two passes alone,
    which grow with n; the forward of 2^14, which one CTA runs in long calls,
    and natural order hold the one-CTA table (8 bytes a coefficient)."""
    two = table_bytes(gb, 4, 16)
    for kind in (4, 5):
        assert table_bytes(gb, kind, 15) * 2 == two
        assert table_bytes(gb, kind, 15, 9) == 8 << 15 and table_bytes(gb, kind, 14, 9) == 8 << 14
    assert table_bytes(gb, 5, 14) * 4 == two
    assert table_bytes(gb, 4, 14) == table_bytes(gb, 5, 14) + (8 << 14)


@pytest.mark.parametrize("L", [14, 15, 16, 18, 20, 22])
def test_two_pass_tables_take_8_bytes_a_coefficient(gb, L):  # noqa: F811
    for kind in (4, 5):
        one_cta = 8 << L if (kind, L) == (4, 14) else 0
        assert table_bytes(gb, kind, L) <= (8 << L) + one_cta
