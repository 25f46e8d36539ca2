/*
 * Places in a buffer that is filled in turn in parts (host): programs and matrices
 * on their way to the device.  A part is left by recording an event behind the
 * copies out of it and entered by waiting for the event of its last use; both
 * happen in one place, whatever made the part full.
 */
#ifndef DK_STAGE_RING_H_
#define DK_STAGE_RING_H_

#include <stddef.h>

namespace dk {

template <size_t PART, int PARTS> struct StageRing {
	int part = 0; /* being filled */
	size_t at = 0; /* bytes of it in use */
	bool used[PARTS] = {}; /* left before: its event has been recorded */

	static constexpr size_t kAlign = 256;

	/* Offset in the buffer of the next `bytes` (at most PART).  `record(p)` marks
	 * the end of part p's copies, `wait(p)` waits for that mark; both return 0 or
	 * a status, which ends the call and leaves the place where it was. */
	template <typename Record, typename Wait>
	int place(size_t bytes, Record record, Wait wait, size_t *offset)
	{
		if (at + bytes > PART) {
			int rc = record(part);
			if (rc)
				return rc;
			used[part] = true;
			const int next = (part + 1) % PARTS;
			if (used[next]) {
				rc = wait(next);
				if (rc)
					return rc;
			}
			part = next;
			at = 0;
		}
		*offset = (size_t)part * PART + at;
		at += (bytes + kAlign - 1) & ~(kAlign - 1);
		return 0;
	}
};

} // namespace dk

#endif
