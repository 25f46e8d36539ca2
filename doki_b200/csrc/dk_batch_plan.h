/*
 * Planning of one batch circuit as factored sweeps (host, used by dk_batch.cu).
 */
#ifndef DK_BATCH_PLAN_H_
#define DK_BATCH_PLAN_H_

#include <vector>

#include "dk_internal.h"

namespace dk {

/* A circuit's programs back to back.  The batch kernels of factored circuits read
 * factored programs and nothing else, without a look at a program's mode. */
struct BatchProgram {
	std::vector<unsigned char> bytes;
	uint32_t nsweep = 0;
	uint32_t most = 0; /* bytes of the longest program */
};

/* 0: planned, or failed with *rc; 1: some step is not a factored sweep (`out` is
 * left empty), the circuit is for the gate-by-gate kernel. */
inline int plan_factored(const std::vector<dk_flat_op> &flat, unsigned n, int prec, int m,
			 BatchProgram *out, int *rc)
{
	dk_plan_limits lim = {};
	lim.tile_bits = m;
	dk_plan_default_limits(prec, n, &lim);
	lim.tile_bits = m;
	dk_fx_plan *fp = nullptr;
	*rc = dk_fx_begin(flat.data(), (int)flat.size(), n, prec, &lim, &fp);
	if (*rc)
		return 0;
	int other = !dk_fx_all(fp);
	int more = 0;
	dk_step step;
	const unsigned char *src;
	while (!other && (more = dk_fx_next(fp, &step, &src)) > 0) {
		const dk_sweep_hdr *h = (const dk_sweep_hdr *)src;
		if (step.kind != 1 || h->mode != DK_SWEEP_FACTORED) {
			other = 1;
			break;
		}
		const uint32_t bytes = h->bytes;
		try {
			out->bytes.insert(out->bytes.end(), src, src + bytes);
		} catch (...) {
			more = -DK_ERR_ALLOC;
			break;
		}
		++out->nsweep;
		if (bytes > out->most)
			out->most = bytes;
	}
	dk_fx_end(fp);
	if (other) {
		out->bytes.clear();
		out->nsweep = out->most = 0;
		return 1;
	}
	*rc = more < 0 ? -more : 0;
	return 0;
}

} // namespace dk

#endif
