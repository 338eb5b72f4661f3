"""A token id that does not fit 32 bits is refused before it reaches the library, which takes an int32."""
import pytest


@pytest.mark.parametrize("token", [2**32 + 5, 2**31, -2**31 - 1])
def test_ids_beyond_32_bits(token):
    import cpmcu.C as C
    with pytest.raises(OverflowError):
        C.decode_token(token, 3, 0, 0, True)
